// Prompt attention on tcgen05 with scores, weights and outputs in tensor memory: causal, varlen, aware of cached positions.
//
//   paged    K/V rows of the token-granular pool, fetched by TMA gathers through the slot table (head size 128)
//   expanded K/V rows of dense matrices formed for the pass (latent attention: key size 192, value size 128 or 64; the last 64 columns
//            of the keys are shared by all heads, see llb_latent_prefill_fa)
//
// A CTA works on two 128-row query tiles against the same keys: two query heads of one KV head where their number is even (paged), else
// 256 consecutive tokens of a head.  Per tile of BN keys and query tile t:
//   S_t  = Q_t . K^T     into tensor memory
//   P_t  = exp2(S_t - m) one thread per row reads its scores, and writes the weights as bf16 over them in tensor memory (expanded form:
//          as the sum of two bf16 values, which makes up for the rounding of the expanded keys and values up to scores of spread 2.5)
//   O_t += P_t . V       A operand from tensor memory, accumulated there over all key tiles
// One thread issues all MMAs in the order  P0.V, Q0.K', P1.V, Q1.K'  so that the tensor core works on one query tile while the softmax
// warps work on the other.  (This schedule, the weights as tensor-memory operand and the rescaling only after the maximum grew by 2^8 were
// published with FlashAttention-4, Dao and others, 2025.)  O is rescaled, read-multiply-write, when a row's maximum has grown: at once where the weights are
// single bf16 values, so that the weight of the largest key is exactly 1 (with a slack of 2^8 it is rounded like the others, and the error
// against 64 bits grew from 0.0018 to 0.0023 for 1000 keys with scores of spread 2.5); by more than 2^8 where they are the sum of two.
//
// What bounds it: per 128 x 128 scores of head size 128, 1024 cycles of MMA and 1024 of exponentials (16 a cycle); it takes about 2100
// (cycle counters without rescaling: softmax 2300 per query tile and key tile, half of it hidden; a warp rescales 128 columns when one of
// its rows' maxima grew).  attention_tc.cu (one query tile, P through shared memory, O in registers, K/V gathered by two warps with 16-byte
// copies, and every MMA's operands moved to uniform registers, see elect_one) needs about 10000.  B200, 32 query and 8 KV heads, scores of
// spread 2, kernel alone at burst clocks: 16 x 1024 tokens 248 us, 8192 tokens 605 us, 4 x 2048 with 4 KV heads 195 us (229, 543 and 178
// with a slack of 2^8; 16 x 1024 took attention_tc.cu 746).
#include "sm100_ptx.cuh"

using namespace llb;
using namespace llb::sm100;
LLB_DEBUG_BOUNDS_STORAGE(attention_fa)

namespace {

constexpr int BM = 128;
constexpr int OWN = 128;          // expanded: key columns of a head's own; the others are shared by all heads
constexpr int THREADS = 12 * 32;  // warp 0: Q and K/V loads (paged: with warps 2, 3), warp 1: MMA, warps 4..7 / 8..11: softmax of query
                                  // tile 0 / 1
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kSlack = 8.f;     // SPLIT_P: log2 of the largest weight before the maximum is moved

__device__ int g_attn_fa_status = 0;  // a wait ran out in some launch, whatever word its caller gave

template <int DK, int DV, int BN>
struct Layout {
  static constexpr int Q_BYTES = DK / 64 * BM * 128, K_BYTES = DK / 64 * BN * 128, V_BYTES = DV / 64 * BN * 128;
  static constexpr int K_SLOTS = 3, V_SLOTS = BN == 128 ? 2 : 3;
  static constexpr int OFF_Q = 0, OFF_K = 2 * Q_BYTES, OFF_V = OFF_K + K_SLOTS * K_BYTES, OFF_BAR = OFF_V + V_SLOTS * V_BYTES;
  static constexpr int BYTES = OFF_BAR + 256;  // the dynamic shared memory starts on a 1024-byte boundary (checked in the kernel)
  static constexpr int S_COL = 0, O_COL = 2 * BN;  // tensor memory: S0 | S1 | O0 | O1
};

struct Params {
  const int *cu_q, *b_ready_len;
  int* status;  // receives the code of a wait that ran out
  bf16* out;
  int64_t out_stride;
  float scale_log2;
  int Hq, Hkv, pairs;  // pairs: the two query tiles are heads 2 y and 2 y + 1 (else tokens 0..127 and 128..255 of head y)
  int n_slots;  // rows of the pool slice, or of the expanded matrix
  // paged
  const int *req_to_token, *b_req_idx;
  int64_t r2t_stride;
  // expanded
  const int *cu_kv, *kv_start;
  int shared_col;
};

__device__ __forceinline__ float ex2_fast(float x) {  // 2^x, one MUFU instruction (x = -inf gives 0)
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// SPLIT_P: the weights enter P . V as high and low part (BN == 64: both fit the columns of the scores)
template <int DK, int DV, int BN, bool PAGED, bool SPLIT_P>
__global__ void __launch_bounds__(THREADS, 1)
prefill_fa_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmKV,
                  const __grid_constant__ CUtensorMap tmShared, const __grid_constant__ CUtensorMap tmRow, const Params p) {
  using L = Layout<DK, DV, BN>;
  static_assert(!SPLIT_P || BN == 64, "the two parts of the weights take the place of the scores");
  constexpr int KS = L::K_SLOTS, VS = L::V_SLOTS;
  extern __shared__ __align__(1024) uint8_t smem[];
  const uint32_t smem_base = smem_u32(smem);
  const uint32_t bar = smem_base + L::OFF_BAR;
  auto k_full = [&](int s) { return bar + 8 * s; };
  auto k_empty = [&](int s) { return bar + 8 * (KS + s); };
  auto v_full = [&](int s) { return bar + 8 * (2 * KS + s); };
  auto v_empty = [&](int s) { return bar + 8 * (2 * KS + VS + s); };
  auto s_full = [&](int t) { return bar + 8 * (2 * KS + 2 * VS + t); };
  auto p_full = [&](int t) { return bar + 8 * (2 * KS + 2 * VS + 2 + t); };
  auto o_full = [&](int t) { return bar + 8 * (2 * KS + 2 * VS + 4 + t); };
  const uint32_t q_full = bar + 8 * (2 * KS + 2 * VS + 6);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + L::OFF_BAR + 200);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + L::OFF_BAR + 204);
  int* status = p.status;

  // heads fastest, late (long) query tiles first
  const int y = blockIdx.x, b = blockIdx.y;
  const int rows_cta = p.pairs ? BM : 2 * BM;
  const int q0 = (int)(gridDim.z - 1 - blockIdx.z) * rows_cta;
  const int q_begin = p.cu_q[b], q_len = p.cu_q[b + 1] - q_begin;
  if (q0 >= q_len) return;  // whole CTA: nothing allocated yet
  if (smem_base & 1023u) {
    if (threadIdx.x == 0) {
      atomicCAS(status, 0, 70);
      g_attn_fa_status = 70;
    }
    return;
  }
  const int ready = p.b_ready_len[b];
  const int kv0 = PAGED ? 0 : p.kv_start[b];
  auto head_of = [&](int t) { return p.pairs ? 2 * y + t : y; };
  auto first_row = [&](int t) { return p.pairs ? q0 : q0 + t * BM; };
  // key tiles that query tile t sees (0: it has no rows)
  auto tiles_of = [&](int t) {
    const int rows = min(BM, q_len - first_row(t));
    return rows > 0 ? (ready + first_row(t) + rows - kv0 + BN - 1) / BN : 0;
  };
  const int n0 = tiles_of(0), n1 = tiles_of(1), n = max(n0, n1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int s = 0; s < KS; ++s) mbar_init(k_full(s), 1), mbar_init(k_empty(s), 1);
    for (int s = 0; s < VS; ++s) mbar_init(v_full(s), 1), mbar_init(v_empty(s), 1);
    for (int t = 0; t < 2; ++t) mbar_init(s_full(t), 1), mbar_init(p_full(t), 4), mbar_init(o_full(t), 1);
    mbar_init(q_full, 1);
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

  if (warp == 0 || (PAGED && (warp == 2 || warp == 3))) {
    // ---- loads ----
    if (warp == 0 && elect_one()) {
      mbar_expect_tx(q_full, (n1 > 0 ? 2 : 1) * L::Q_BYTES);
      for (int t = 0; t < (n1 > 0 ? 2 : 1); ++t)
#pragma unroll
        for (int c = 0; c < DK / 64; ++c)
          tma_load_2d(smem_base + L::OFF_Q + t * L::Q_BYTES + c * BM * 128, &tmQ, q_full, head_of(t) * DK + c * 64,
                      q_begin + first_row(t));
    }
    __syncwarp();
    if (PAGED) {
      // A gather costs its warp about 70 cycles to issue (every lane's operands go through the uniform registers), 128 of them per tile:
      // the three warps take the gathers of four keys in turn
      const int kv_end = ready + min(q_len, q0 + rows_cta);  // exclusive bound on the keys any row sees
      const int* table = p.req_to_token + (int64_t)LLB_CHECK_REQ(p.b_req_idx[b]) * p.r2t_stride;
      const int kvh = head_of(0) / (p.Hq / p.Hkv);
      const int k_col = kvh * DK, v_col = p.Hkv * DK + kvh * DV;
      const int quad = lane * 3 + (warp == 0 ? 0 : warp - 1);  // keys 4 quad .. 4 quad + 3 of a tile
      const bool active = quad < BN / 4;
      int next[4];
      auto fetch = [&](int j) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int pos = j * BN + quad * 4 + e;
          next[e] = active && pos < kv_end ? LLB_CHECK_SLOT(table[pos]) : p.n_slots;  // row n_slots: out of range, reads zeros
        }
      };
      fetch(0);
      for (int j = 0; j < n; ++j) {
        const int ks = j % KS, vs = j % VS;
        const int r0 = next[0], r1 = next[1], r2 = next[2], r3 = next[3];
        if (j + 1 < n) fetch(j + 1);
        if (!__all_sync(0xffffffffu, mbar_wait(k_empty(ks), ((j / KS) & 1) ^ 1, abort_flag, status, 71))) break;
        if (warp == 0 && lane == 0) mbar_expect_tx(k_full(ks), L::K_BYTES);
        if (active)
#pragma unroll
          for (int c = 0; c < DK / 64; ++c)
            tma_gather4(smem_base + L::OFF_K + ks * L::K_BYTES + c * BN * 128 + quad * 512, &tmKV, k_full(ks), k_col + c * 64, r0, r1,
                        r2, r3);
        __syncwarp();
        if (!__all_sync(0xffffffffu, mbar_wait(v_empty(vs), ((j / VS) & 1) ^ 1, abort_flag, status, 72))) break;
        if (warp == 0 && lane == 0) mbar_expect_tx(v_full(vs), L::V_BYTES);
        if (active)
#pragma unroll
          for (int c = 0; c < DV / 64; ++c)
            tma_gather4(smem_base + L::OFF_V + vs * L::V_BYTES + c * BN * 128 + quad * 512, &tmKV, v_full(vs), v_col + c * 64, r0, r1,
                        r2, r3);
        __syncwarp();
      }
    } else if (elect_one()) {
      // The rows behind a request's last one are its neighbour's first.  Their scores are masked, but a weight of 0 times a value that
      // is not finite is not 0: the values of the tile that holds the end come row by row, zeros in the place of the others.
      const int row0 = p.cu_kv[b], rows = ready + q_len - kv0;
      for (int j = 0; j < n; ++j) {
        const int ks = j % KS, vs = j % VS;
        if (!mbar_wait(k_empty(ks), ((j / KS) & 1) ^ 1, abort_flag, status, 71)) break;
        mbar_expect_tx(k_full(ks), L::K_BYTES);
#pragma unroll
        for (int c = 0; c < DK / 64; ++c) {
          const bool mine = c * 64 < OWN;
          tma_load_2d(smem_base + L::OFF_K + ks * L::K_BYTES + c * BN * 128, mine ? &tmKV : &tmShared, k_full(ks),
                      mine ? y * OWN + c * 64 : p.shared_col + c * 64 - OWN, row0 + j * BN);
        }
        if (!mbar_wait(v_empty(vs), ((j / VS) & 1) ^ 1, abort_flag, status, 72)) break;
        mbar_expect_tx(v_full(vs), L::V_BYTES);
        const uint32_t v = smem_base + L::OFF_V + vs * L::V_BYTES;
        const int v_col = p.Hq * OWN + y * DV;
        if ((j + 1) * BN <= rows) {
#pragma unroll
          for (int c = 0; c < DV / 64; ++c) tma_load_2d(v + c * BN * 128, &tmKV, v_full(vs), v_col + c * 64, row0 + j * BN);
        } else {
#pragma unroll 1
          for (int i = j * BN; i < (j + 1) * BN; i += 4) {
            auto row = [&](int e) { return i + e < rows ? row0 + i + e : p.n_slots; };  // row n_slots: out of range, reads zeros
#pragma unroll
            for (int c = 0; c < DV / 64; ++c)
              tma_gather4(v + c * BN * 128 + (i - j * BN) * 128, &tmRow, v_full(vs), v_col + c * 64, row(0), row(1), row(2), row(3));
          }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (elect_one()) {
      // ---- MMA issuer.  MMAs of one thread run in the order they are issued, so S_t of the next tile, which overwrites P_t, may be
      // issued right behind P_t . V ----
      constexpr uint32_t IDESC_S = umma_idesc(BM, BN, 1);
      constexpr uint32_t IDESC_PV = umma_idesc(BM, 64, 1) | (1u << 16);  // B operand MN-major
      auto scores = [&](int t, int j) {
        const uint32_t q = smem_base + L::OFF_Q + t * L::Q_BYTES, k = smem_base + L::OFF_K + (j % KS) * L::K_BYTES;
        if (!mbar_wait(k_full(j % KS), (j / KS) & 1, abort_flag, status, 73)) return false;
        tc_fence_after();
        const uint64_t dq = umma_smem_desc_sw128(q), dk = umma_smem_desc_sw128(k);  // offsets count 16-byte units
#pragma unroll
        for (int i = 0; i < DK / 16; ++i)
          umma_bf16(tmem_base + L::S_COL + t * BN, dq + ((i >> 2) * BM * 8 + (i & 3) * 2), dk + ((i >> 2) * BN * 8 + (i & 3) * 2),
                    IDESC_S, i != 0);
        umma_commit(s_full(t));
        return true;
      };
      auto values = [&](int t, int j) {
        const uint32_t v = smem_base + L::OFF_V + (j % VS) * L::V_BYTES;
        if (!mbar_wait(p_full(t), j & 1, abort_flag, status, 74) || !mbar_wait(v_full(j % VS), (j / VS) & 1, abort_flag, status, 75)) return false;
        tc_fence_after();
        const uint64_t dv = umma_smem_desc_sw128_mn(v);
#pragma unroll
        for (int h = 0; h < DV / 64; ++h)
#pragma unroll
          for (int i = 0; i < (SPLIT_P ? 2 : 1) * BN / 16; ++i)
            umma_bf16_ts(tmem_base + L::O_COL + t * DV + h * 64, tmem_base + L::S_COL + t * BN + i * 8,
                         dv + (h * BN * 8 + i % (BN / 16) * 128), IDESC_PV, (j | i) != 0);
        umma_commit(o_full(t));
        return true;
      };
      // the second query tile sees at least the key tiles of the first, or has no rows
      bool ok = mbar_wait(q_full, 0, abort_flag, status, 76) && scores(0, 0) && (n1 == 0 || scores(1, 0));  // false: issue nothing more
      if (ok) umma_commit(k_empty(0));
      for (int j = 0; j < n && ok; ++j) {
        const bool k_next = j + 1 < n;
        if (j < n0) ok = values(0, j) && (j + 1 >= n0 || scores(0, j + 1));
        if (ok && j < n1) ok = values(1, j) && (j + 1 >= n1 || scores(1, j + 1));
        if (!ok) break;
        umma_commit(v_empty(j % VS));
        if (k_next) umma_commit(k_empty((j + 1) % KS));
      }
    }
    __syncwarp();
  } else if (warp >= 4) {
    // ---- softmax: one thread per query row ----
    const int t = (warp - 4) >> 2, lane_grp = warp & 3;
    const int mine = t == 0 ? n0 : n1;
    if (mine > 0) {
      const int row = lane_grp * 32 + lane, tok = first_row(t) + row;
      const int last = min(ready + tok, ready + q_len - 1) - kv0;  // last key this row sees, counted from the first one
      const uint32_t t_lane = tmem_base + ((uint32_t)(lane_grp * 32) << 16);
      const uint32_t t_s = t_lane + L::S_COL + t * BN, t_o = t_lane + L::O_COL + t * DV;
      float m = -INFINITY, l = 0.f;
      for (int j = 0; j < mine; ++j) {
        if (!__all_sync(0xffffffffu, mbar_wait(s_full(t), j & 1, abort_flag, status, 77))) break;
        tc_fence_after();
        uint32_t s[BN];
#pragma unroll
        for (int c = 0; c < BN; c += 32) tmem_ld_32x32(t_s + c, s + c);
#pragma unroll
        for (int c = 0; c < BN; c += 16) tmem_wait_ld_of(s + c);
        const int lim = last - j * BN;  // columns 0 .. lim are seen
        if (lim < BN - 1) {             // only tiles at the diagonal and the end
#pragma unroll
          for (int c = 0; c < BN; ++c)
            if (c > lim) s[c] = 0xff800000u;
        }
        float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int c = 0; c < BN; ++c) mx[c & 3] = fmaxf(mx[c & 3], __uint_as_float(s[c]));
        const float top = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * p.scale_log2;
        const bool moved = top > m + (SPLIT_P ? kSlack : 0.f) || m == -INFINITY;
        if (__any_sync(0xffffffffu, moved)) {
          const float m_new = moved ? fmaxf(m, top) : m;
          if (j > 0) {  // O holds the tiles before this one
            const float alpha = m_new == m ? 1.f : ex2_fast(m - m_new);
            l *= alpha;
            mbar_wait(o_full(t), (j - 1) & 1, abort_flag, status, 78);
            tc_fence_after();
            tmem_scale<DV>(t_o, alpha);
          }
          m = m_new;
        }
        const float base = m == -INFINITY ? 0.f : m;
        float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int h = 0; h < BN / 64; ++h) {
          uint32_t w[32], low[32];
#pragma unroll
          for (int c = 0; c < 32; ++c) {
            const float a = ex2_fast(fmaf(__uint_as_float(s[h * 64 + 2 * c]), p.scale_log2, -base));
            const float d = ex2_fast(fmaf(__uint_as_float(s[h * 64 + 2 * c + 1]), p.scale_log2, -base));
            sum[(2 * c) & 3] += a;
            sum[(2 * c + 1) & 3] += d;
            w[c] = pack_bf16x2(a, d);
            if (SPLIT_P) low[c] = pack_bf16x2(a - __uint_as_float(w[c] << 16), d - __uint_as_float(w[c] & 0xffff0000u));
          }
          tmem_st_32x32(t_s + h * 32, w);
          if (SPLIT_P) tmem_st_32x32(t_s + 32, low);
        }
        l += (sum[0] + sum[1]) + (sum[2] + sum[3]);
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(p_full(t));
      }
      const bool whole = __all_sync(0xffffffffu, mbar_wait(o_full(t), (mine - 1) & 1, abort_flag, status, 79)) && !*abort_flag;
      tc_fence_after();
      // output: a warp parks its 32 rows in the (now idle) query tile and writes whole rows
      const float inv = l > 0.f ? 1.f / l : 0.f;
      uint8_t* stg = smem + L::OFF_Q + t * L::Q_BYTES + lane_grp * 32 * (DV * 2);
      constexpr int CH = DV / 8;  // 16-byte chunks of a row
#pragma unroll
      for (int c = 0; c < DV; c += 32) {
        uint32_t r[32];
        tmem_ld_32x32(t_o + c, r);
        tmem_wait_ld_of(r);
        tmem_wait_ld_of(r + 16);
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          float v[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) v[e] = __uint_as_float(r[g * 8 + e]) * inv;
          *reinterpret_cast<bf16x8*>(stg + lane * (DV * 2) + (((c / 8 + g) ^ (lane & 7)) << 4)) = pack8(v);
        }
      }
      __syncwarp();
#pragma unroll 4
      for (int i = 0; i < CH; ++i) {
        const int id = i * 32 + lane, r = id / CH, ch = id % CH;
        const int tk = first_row(t) + lane_grp * 32 + r;
        if (tk < q_len && whole)
          *reinterpret_cast<bf16x8*>(p.out + (int64_t)(q_begin + tk) * p.out_stride + head_of(t) * DV + ch * 8) =
              *reinterpret_cast<const bf16x8*>(stg + r * (DV * 2) + ((ch ^ (r & 7)) << 4));
      }
      tc_fence_before();
    }
  }

  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    settle_after_abort();
    if (threadIdx.x == 0) g_attn_fa_status = 1;
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

template <int DK, int DV, int BN, bool PAGED, bool SPLIT_P>
int launch_fa(const CUtensorMap& tq, const CUtensorMap& tkv, const CUtensorMap& ts, const CUtensorMap& trow, const Params& p, int B,
              int max_q_len, cudaStream_t st) {
  using L = Layout<DK, DV, BN>;
  static_assert(L::BYTES <= 227 * 1024, "shared memory");
  static_assert(2 * BN + 2 * DV <= 512, "tensor memory");
  static_assert((2 * L::K_SLOTS + 2 * L::V_SLOTS + 7) * 8 <= 200, "barriers");
  static DeviceOnce configured;
  if (!configured.done()) {
    cudaError_t e = cudaFuncSetAttribute(prefill_fa_kernel<DK, DV, BN, PAGED, SPLIT_P>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, L::BYTES);
    if (e != cudaSuccess) return (int)e;
    configured.set();
  }
  const int rows = p.pairs ? BM : 2 * BM;
  prefill_fa_kernel<DK, DV, BN, PAGED, SPLIT_P>
      <<<dim3(p.pairs ? p.Hq / 2 : p.Hq, B, cdiv(max_q_len, rows)), THREADS, L::BYTES, st>>>(tq, tkv, ts, trow, p);
  LLB_LAUNCH_CHECK();
  return LLB_OK;
}

}  // namespace

// 0 while every bounded wait of the kernel was met; 70: shared memory not where the layout needs it; 1: a wait ran out (its code is in
// the status word of that launch).
LLB_EXPORT int llb_attn_fa_status() {
  int v = 0;
  cudaMemcpyFromSymbol(&v, g_attn_fa_status, sizeof(int));
  return v;
}

// Same contract as llb_gqa_prefill with head size 128; T rows of q, n_slots rows of the pool slice; status: device int that receives the
// code of a wait that ran out.
LLB_EXPORT int llb_gqa_prefill_fa(const void* q, int64_t q_stride, int T, const void* kv_layer, int n_slots, const int* req_to_token,
                                  int64_t r2t_stride, const int* b_req_idx, const int* cu_q, const int* b_ready_len, void* out,
                                  int64_t out_stride, int B, int max_q_len, int Hq, int Hkv, float sm_scale, int* status, cudaStream_t st) {
  if (B <= 0 || max_q_len <= 0 || T <= 0) return LLB_OK;
  if (!(sm_scale > 0.f) || status == nullptr || Hkv <= 0 || Hq % Hkv != 0 || n_slots <= 0 || (out_stride % 8) || ((uintptr_t)out & 15)) return LLB_ERR_BAD_ARG;
  if (B > 65535 || cdiv(max_q_len, BM) > 65535) return LLB_ERR_UNSUPPORTED;
  CUtensorMap tq, tkv;
  int rc = make_tmap_2d(&tq, q, 2, (uint64_t)T, (uint64_t)Hq * 128, (uint64_t)q_stride, BM, 64);
  if (rc) return rc;
  rc = make_tmap_2d(&tkv, kv_layer, 2, (uint64_t)n_slots, (uint64_t)Hkv * 256, (uint64_t)Hkv * 256, 1, 64);
  if (rc) return rc;
  Params p;
  memset(&p, 0, sizeof(p));
  p.status = status, p.cu_q = cu_q, p.b_ready_len = b_ready_len, p.out = (bf16*)out, p.out_stride = out_stride, p.scale_log2 = sm_scale * kLog2e;
  p.Hq = Hq, p.Hkv = Hkv, p.pairs = (Hq / Hkv) % 2 == 0;
  p.req_to_token = req_to_token, p.b_req_idx = b_req_idx, p.r2t_stride = r2t_stride, p.n_slots = n_slots;
  return launch_fa<128, 128, 128, true, false>(tq, tkv, tkv, tkv, p, B, max_q_len, st);
}

// q [T, >= H * 192] bf16 (row pitch q_stride), kv [kv_rows, H * 128 | H * dv] (pitch kv_stride), out [T, >= H * dv].  Request b's
// keys are rows cu_kv[b] .., position kv_start[b] first; the last 64 columns of every head's keys are columns shared_col .. of `shared`
// [kv_rows, >= shared_col + 64] (pitch shared_stride).
LLB_EXPORT int llb_latent_prefill_fa(const void* q, int64_t q_stride, const void* kv, int64_t kv_stride, int kv_rows,
                                     const void* shared, int64_t shared_stride, int shared_col, const int* cu_q,
                                     const int* cu_kv, const int* kv_start, const int* b_ready_len, void* out, int64_t out_stride,
                                     int B, int T, int max_q_len, int H, int dv, float sm_scale, int* status, cudaStream_t st) {
  if (B <= 0 || max_q_len <= 0 || T <= 0) return LLB_OK;
  if (!(sm_scale > 0.f) || status == nullptr || H <= 0 || kv_rows <= 0 || (out_stride % 8) || ((uintptr_t)out & 15)) return LLB_ERR_BAD_ARG;
  if (B > 65535 || cdiv(max_q_len, BM) > 65535 || (dv != 64 && dv != 128)) return LLB_ERR_UNSUPPORTED;
  if (shared == nullptr || shared_col < 0 || (shared_col % 8)) return LLB_ERR_BAD_ARG;
  CUtensorMap tq, tkv, ts, trow;
  int rc = make_tmap_2d(&tq, q, 2, (uint64_t)T, (uint64_t)H * 192, (uint64_t)q_stride, BM, 64);
  if (rc) return rc;
  rc = make_tmap_2d(&tkv, kv, 2, (uint64_t)kv_rows, (uint64_t)H * (OWN + dv), (uint64_t)kv_stride, 64, 64);
  if (rc) return rc;
  rc = make_tmap_2d(&trow, kv, 2, (uint64_t)kv_rows, (uint64_t)H * (OWN + dv), (uint64_t)kv_stride, 1, 64);
  if (rc) return rc;
  rc = make_tmap_2d(&ts, shared, 2, (uint64_t)kv_rows, (uint64_t)shared_col + 64, (uint64_t)shared_stride, 64, 64);
  if (rc) return rc;
  Params p;
  memset(&p, 0, sizeof(p));
  p.status = status, p.cu_q = cu_q, p.b_ready_len = b_ready_len, p.out = (bf16*)out, p.out_stride = out_stride, p.scale_log2 = sm_scale * kLog2e;
  p.Hq = p.Hkv = H, p.n_slots = kv_rows, p.cu_kv = cu_kv, p.kv_start = kv_start, p.shared_col = shared_col;
  return dv == 64 ? launch_fa<192, 64, 64, false, true>(tq, tkv, ts, trow, p, B, max_q_len, st)
                  : launch_fa<192, 128, 64, false, true>(tq, tkv, ts, trow, p, B, max_q_len, st);
}
