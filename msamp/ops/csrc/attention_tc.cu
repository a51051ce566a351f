// Softmax attention for bf16, head sizes 64 and 128, on the sm_100a tensor path (tcgen05 + TMEM + TMA).
//
// The kernels share one structure: one warp streams operand tiles with TMA (4-D tensor maps over the strided
// [batch, seq, head, head_dim] views, 128-byte swizzle), one or two warps issue tcgen05.mma (kind::f16) into TMEM, and two
// groups of four warps (one thread per accumulator row) read the scores back with tcgen05.ld, do the softmax arithmetic and
// write the bf16 operand of the next MMA into TMEM or into swizzled shared memory.
//
//   attn_fwd_ps_kernel        forward, 128 queries x 128 keys per tile: S = Q K^T  ->  P = exp2(S - m)  ->  O += P V
//   attn_bwd_dkdv_ps_kernel   128 key rows: S^T = K Q^T, dP^T = V dO^T, dV += P^T dO, dK += dS^T Q
//   attn_bwd_dq_ps_kernel     128 query rows: S = Q K^T, dP = dO V^T, dQ += dS K
//   attn_fwd_tm_kernel, attn_fwd_split_kernel   forward of short rows of head size 128, two maxima per row (see kSplitRows)
// Head size 128 also has earlier kernels with one CTA per work item, and with 64-wide tiles and P / dS in shared memory; they
// run when MSAMP_ATTN_{FWD,BWD}_PERSIST=0 or MSAMP_ATTN_{FWD,BWD}_SMEM=1 and serve as a cross-check.
//
// V, dO, Q and K enter the second kind of product with the reduction index as rows of the tile, so
// the same shared-memory tile is described once K-major and once MN-major; nothing is transposed.
// The backward pass is deterministic (no atomics).  Every mbarrier wait is bounded; when one gives
// up, bit 2 (value 4) of the device status word is set and the CTA frees its TMEM and returns.
//
// Head size 64 took the mma.sync kernels of attention.cu before: 8 x 1024 x 12 heads, causal, 71 + 253 us forward + backward on
// the device, now 44 + 107 us; 64 x 197 x 12 heads, 61 + 218 us, now 45 + 119 us.  Those kernels remain for views that a tensor map
// cannot describe, for short rows (see short_rows) and as a cross-check (MSAMP_ATTN_IMPL=mma).
#include <cstdlib>
#include <mutex>
#include <unordered_map>

#include "tcgen05.cuh"

namespace {

constexpr int kTcThreads = 320;    // warp 0: TMA, warp 1: MMA, warps 2-5 and 6-9: the two softmax groups
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;
constexpr unsigned int kStatusBit = 4u;

struct TcParams {
  __nv_bfloat16* o;
  float* lse;             // [b, h, s] natural-log sum-exp of the scaled scores
  const float* delta;     // [b, h, s] rowsum(dO * O)
  __nv_bfloat16* dq;
  __nv_bfloat16* dk;
  __nv_bfloat16* dv;
  int64_t o_sb, o_ss, o_sh;    // element strides: batch, sequence, head
  int64_t dq_sb, dq_ss, dq_sh;
  int64_t dk_sb, dk_ss, dk_sh;
  int64_t dv_sb, dv_ss, dv_sh;
  int batch, heads, seqlen, causal;
  int group;              // persistent kernels: (batch, head) pairs whose work items are taken together
  float scale;
  unsigned int* status;
};

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  __nv_bfloat162 t = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&t);
}
__device__ __forceinline__ void st_shared_v4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
// Columns i > last of a 64-column slice become `v` (the masked end of a diagonal or ragged tile).
__device__ __forceinline__ void mask_above(uint32_t (&r)[2][32], int last, uint32_t v) {
#pragma unroll
  for (int i = 0; i < 64; ++i)
    if (i > last) r[i >> 5][i & 31] = v;
}

// Makes this thread's ordinary shared-memory writes visible to the async proxy (the MMA reads them).
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// 128 fp32 values of one row -> bf16 -> 256 contiguous bytes in global memory.
__device__ __forceinline__ void st_row32(__nv_bfloat16* dst, const float (&v)[32]) {
  uint4* d4 = reinterpret_cast<uint4*>(dst);
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    uint4 u;
    u.x = pack_bf16(v[8 * t], v[8 * t + 1]);
    u.y = pack_bf16(v[8 * t + 2], v[8 * t + 3]);
    u.z = pack_bf16(v[8 * t + 4], v[8 * t + 5]);
    u.w = pack_bf16(v[8 * t + 6], v[8 * t + 7]);
    d4[t] = u;
  }
}

// Stores 64 columns of the 32 rows of a warp, one row per lane on entry.  A row of 64 bf16 is eight 16-byte chunks: an 8 x 8
// transposition of chunks inside every eight lanes (three butterfly steps) turns "one row per lane" into "one chunk of eight
// rows per lane", so that every store instruction writes four whole 128-byte lines.  With one row per lane it wrote 32
// half-used sectors, and the epilogue of a dK / dV item took 7700 cycles of some 40000.
__device__ __forceinline__ void st_rows64(__nv_bfloat16* dst, int64_t stride, int rows, const float (&v)[64]) {
  const int lane = threadIdx.x & 31;
  uint32_t x[8][4];
#pragma unroll
  for (int c = 0; c < 8; ++c)
#pragma unroll
    for (int k = 0; k < 4; ++k) x[c][k] = pack_bf16(v[8 * c + 2 * k], v[8 * c + 2 * k + 1]);
#pragma unroll
  for (int s = 1; s < 8; s <<= 1) {
    const bool up = (lane & s) != 0;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      if (c & s) continue;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const uint32_t got = __shfl_xor_sync(0xffffffffu, up ? x[c][k] : x[c | s][k], s);
        if (up) x[c][k] = got;
        else    x[c | s][k] = got;
      }
    }
  }
  const int r0 = lane & ~7;
#pragma unroll
  for (int i = 0; i < 8; ++i)
    if (r0 + i < rows) *reinterpret_cast<uint4*>(dst + (int64_t)(r0 + i) * stride + (lane & 7) * 8) = make_uint4(x[i][0], x[i][1], x[i][2], x[i][3]);
}

#define TC_WAIT(bar_, ph_) \
  if (!tc5::mbar_wait((bar_), (ph_), abort_flag, p.status, kStatusBit)) break

// ============================================================================================ forward
namespace fwd {
constexpr int NB = 4;                         // ring depth of the K, V, S and P buffers (key tile j uses slot j & 3)
constexpr uint32_t PANEL_Q = 128 * 128;       // [128 query rows][64 bf16]
constexpr uint32_t TILE_Q = 2 * PANEL_Q;
constexpr uint32_t PANEL_KV = 64 * 128;       // [64 key rows][64 bf16]
constexpr uint32_t TILE_KV = 2 * PANEL_KV;    // 16 KB
constexpr uint32_t TILE_P = 128 * 128;        // [128 query rows][64 keys] bf16
constexpr uint32_t OFF_Q = 0, OFF_K = TILE_Q, OFF_V = OFF_K + NB * TILE_KV, OFF_P = OFF_V + NB * TILE_KV, OFF_BAR = OFF_P + NB * TILE_P;
enum { B_Q = 0, B_KF = 1, B_KE = B_KF + NB, B_VF = B_KE + NB, B_VE = B_VF + NB, B_SF = B_VE + NB, B_SE = B_SF + NB, B_PF = B_SE + NB,
       B_PE = B_PF + NB, B_OF = B_PE + NB, B_ACC = B_OF + 2, NBAR = B_ACC + 1 };
constexpr int SMEM = OFF_BAR + NBAR * 8 + 16 + 1024;
constexpr uint32_t TM_S = 0, TM_O = 256, TM_COLS = 512;    // four 64-column score buffers, two 128-column outputs
constexpr float kRescaleStep = 8.0f;    // the reference maximum may lag the true one by 2^8
}    // namespace fwd

// The two softmax groups work on alternating key tiles (64 keys each) and never exchange anything
// inside the loop: group g owns the score and probability slots of its tiles and its own output
// accumulator O_g in TMEM with its own reference maximum m_g and row sum l_g, i.e. each group computes
// attention over its half of the key tiles and the halves are merged once at the end.  Scores are
// computed up to four tiles ahead, so a group finds its next S ready when it has finished a tile.
// O_g stays in TMEM and is accumulated by the MMA itself; it is only read back and rescaled when a
// row's maximum grew by more than kRescaleStep since the last rescale (probabilities then stay
// below 2^8, far inside bf16/fp32 range).
__global__ void __launch_bounds__(kTcThreads, 1)
attn_fwd_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                   const __grid_constant__ CUtensorMap map_v, const TcParams p) {
  using namespace fwd;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = tc5::smem_u32(smem_raw);
  const uint32_t base = (raw_addr + 1023u) & ~1023u;
  uint8_t* smem = smem_raw + (base - raw_addr);
  const uint32_t bars = base + OFF_BAR;
  auto bar = [&](int i) { return bars + 8u * (uint32_t)i; };
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(smem + OFF_BAR + NBAR * 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);
  // Wait used by full warps that go on to warp-collective TMEM accesses: the outcome is made uniform.
  auto wait_warp = [&](uint32_t br, uint32_t ph) {
    return __all_sync(0xffffffffu, tc5::mbar_wait(br, ph, abort_flag, p.status, kStatusBit)) != 0;
  };

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int qt = (int)gridDim.x - 1 - (int)blockIdx.x;    // long rows first
  const int bh = blockIdx.y;
  const int b = bh / p.heads;
  const int h = bh - b * p.heads;
  const int q0 = qt * 128;
  const int n_all = (p.seqlen + 63) / 64;
  const int n_kv = p.causal ? min(2 * qt + 2, n_all) : n_all;

  if (threadIdx.x == 0) {
    tc5::mbar_init(bar(B_Q), 1);
    for (int s = 0; s < NB; ++s) {
      tc5::mbar_init(bar(B_KF + s), 1);
      tc5::mbar_init(bar(B_KE + s), 1);
      tc5::mbar_init(bar(B_VF + s), 1);
      tc5::mbar_init(bar(B_VE + s), 1);
      tc5::mbar_init(bar(B_SF + s), 1);
      tc5::mbar_init(bar(B_SE + s), 4);
      tc5::mbar_init(bar(B_PF + s), 4);
      tc5::mbar_init(bar(B_PE + s), 1);
    }
    tc5::mbar_init(bar(B_OF + 0), 1);
    tc5::mbar_init(bar(B_OF + 1), 1);
    tc5::mbar_init(bar(B_ACC), 1);
    *abort_flag = 0;
    tc5::mbar_fence_init();
    tc5::tma_prefetch_desc(&map_q);
    tc5::tma_prefetch_desc(&map_k);
    tc5::tma_prefetch_desc(&map_v);
  }
  if (warp == 1) {
    tc5::tmem_alloc(tc5::smem_u32(tmem_holder), TM_COLS);
    tc5::tmem_relinquish();
  }
  tc5::fence_before_sync();
  __syncthreads();
  tc5::fence_after_sync();
  const uint32_t tmem_base = *tmem_holder;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      tc5::mbar_arrive_expect_tx(bar(B_Q), TILE_Q);
      tc5::tma_load_4d(base + OFF_Q, &map_q, 0, h, q0, b, bar(B_Q));
      tc5::tma_load_4d(base + OFF_Q + PANEL_Q, &map_q, 64, h, q0, b, bar(B_Q));
      for (int j = 0; j < n_kv; ++j) {
        const int s = j & (NB - 1);
        const uint32_t ph = (uint32_t)(j / NB) & 1u;
        TC_WAIT(bar(B_KE + s), ph ^ 1u);
        tc5::mbar_arrive_expect_tx(bar(B_KF + s), TILE_KV);
        tc5::tma_load_4d(base + OFF_K + s * TILE_KV, &map_k, 0, h, j * 64, b, bar(B_KF + s));
        tc5::tma_load_4d(base + OFF_K + s * TILE_KV + PANEL_KV, &map_k, 64, h, j * 64, b, bar(B_KF + s));
        TC_WAIT(bar(B_VE + s), ph ^ 1u);
        tc5::mbar_arrive_expect_tx(bar(B_VF + s), TILE_KV);
        tc5::tma_load_4d(base + OFF_V + s * TILE_KV, &map_v, 0, h, j * 64, b, bar(B_VF + s));
        tc5::tma_load_4d(base + OFF_V + s * TILE_KV + PANEL_KV, &map_v, 64, h, j * 64, b, bar(B_VF + s));
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (lane == 0) {
      const uint32_t idesc_s = tc5::idesc_bf16(128, 64, 0, 0);
      const uint32_t idesc_o = tc5::idesc_bf16(128, 128, 0, 1);
      // S[j&3] = Q K_j^T
      auto issue_s = [&](int j) -> bool {
        const int s = j & (NB - 1);
        const uint32_t ph = (uint32_t)(j / NB) & 1u;
        if (!tc5::mbar_wait(bar(B_SE + s), ph ^ 1u, abort_flag, p.status, kStatusBit)) return false;
        if (!tc5::mbar_wait(bar(B_KF + s), ph, abort_flag, p.status, kStatusBit)) return false;
        tc5::fence_after_sync();
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
          const uint32_t offa = (uint32_t)(kk >> 2) * PANEL_Q + (uint32_t)(kk & 3) * 32u;
          const uint32_t offb = (uint32_t)(kk >> 2) * PANEL_KV + (uint32_t)(kk & 3) * 32u;
          tc5::mma_f16(tmem_base + TM_S + (uint32_t)s * 64u, tc5::smem_desc_k_sw128(base + OFF_Q + offa),
                       tc5::smem_desc_k_sw128(base + OFF_K + s * TILE_KV + offb), idesc_s, kk ? 1u : 0u);
        }
        tc5::mma_commit(bar(B_KE + s));
        tc5::mma_commit(bar(B_SF + s));
        return true;
      };
      do {
        TC_WAIT(bar(B_Q), 0u);
        bool ok = true;
        for (int j = 0; j < NB && j < n_kv; ++j)
          if (!issue_s(j)) { ok = false; break; }
        if (!ok) break;
        for (int j = 0; j < n_kv; ++j) {
          const int s = j & (NB - 1);
          const uint32_t ph = (uint32_t)(j / NB) & 1u;
          if (!tc5::mbar_wait(bar(B_PF + s), ph, abort_flag, p.status, kStatusBit)) { ok = false; break; }
          if (!tc5::mbar_wait(bar(B_VF + s), ph, abort_flag, p.status, kStatusBit)) { ok = false; break; }
          tc5::fence_after_sync();
          // O[j&1] (+)= P_j V_j : A = P (K-major), B = V with the key index as rows (MN-major)
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) {
            tc5::mma_f16(tmem_base + TM_O + (uint32_t)(j & 1) * 128u, tc5::smem_desc_k_sw128(base + OFF_P + s * TILE_P + (uint32_t)kk * 32u),
                         tc5::smem_desc_mn_sw128(base + OFF_V + s * TILE_KV + (uint32_t)kk * 2048u, PANEL_KV), idesc_o,
                         (j >= 2 || kk) ? 1u : 0u);
          }
          tc5::mma_commit(bar(B_VE + s));
          tc5::mma_commit(bar(B_PE + s));
          tc5::mma_commit(bar(B_OF + (j & 1)));
          if (j + NB < n_kv && !issue_s(j + NB)) { ok = false; break; }
        }
        if (ok) tc5::mma_commit(bar(B_ACC));
      } while (false);
    }
  } else {
    // ------------------------------------------------------------------ softmax: one thread per query row and group
    const int qd = warp & 3;           // TMEM lane quarter this warp may access
    const int wg = (warp - 2) >> 2;    // group 0: even key tiles, group 1: odd key tiles
    const int row = qd * 32 + lane;
    const int grow = q0 + row;
    const uint32_t tlane = tmem_base + ((uint32_t)(qd * 32) << 16);
    const uint32_t to = tlane + TM_O + (uint32_t)wg * 128u;
    const float sl = p.scale * kLog2e;
    const int lim = p.causal ? min(grow, p.seqlen - 1) : p.seqlen - 1;    // last visible column
    const uint32_t swz = (uint32_t)(row & 7);
    float m = -INFINITY, l = 0.0f;    // reference maximum (log2 units) and row sum of this group
    bool ok = true;

    for (int j = wg; j < n_kv; j += 2) {
      const int s = j & (NB - 1);
      const uint32_t ph = (uint32_t)(j / NB) & 1u;
      const int k = j >> 1;    // index of this tile within the group
      if (!wait_warp(bar(B_SF + s), ph)) { ok = false; break; }
      tc5::fence_after_sync();
      uint32_t r[2][32];
      tc5::tmem_ld32(tlane + TM_S + (uint32_t)s * 64u, r[0]);
      tc5::tmem_ld32(tlane + TM_S + (uint32_t)s * 64u + 32u, r[1]);
      tc5::tmem_ld_wait();
      tc5::fence_before_sync();
      __syncwarp();
      if (lane == 0) tc5::mbar_arrive(bar(B_SE + s));    // the slot may take the scores of tile j + 4
      const int col0 = j * 64;
      const bool need_mask = (p.causal && col0 + 63 > q0) || (col0 + 64 > p.seqlen);
      float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
      if (need_mask) {
#pragma unroll
        for (int i = 0; i < 64; ++i)
          if (col0 + i <= lim) mx4[i & 3] = fmaxf(mx4[i & 3], __uint_as_float(r[i >> 5][i & 31]));
      } else {
#pragma unroll
        for (int i = 0; i < 64; ++i) mx4[i & 3] = fmaxf(mx4[i & 3], __uint_as_float(r[i >> 5][i & 31]));
      }
      const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * sl;    // sl > 0
      const bool grow_m = mx > m + kRescaleStep || (m == -INFINITY && mx > -INFINITY);
      if (__any_sync(0xffffffffu, grow_m)) {
        const float m_new = grow_m ? mx : m;
        const float corr = (m == -INFINITY) ? 0.0f : ex2(m - m_new);
        if (k > 0) {
          // every earlier product of this group must have landed in O before it is rescaled
          if (!wait_warp(bar(B_OF + wg), (uint32_t)(k - 1) & 1u)) { ok = false; break; }
          tc5::fence_after_sync();
#pragma unroll 1
          for (int c = 0; c < 4; ++c) {
            uint32_t x[32];
            tc5::tmem_ld32(to + (uint32_t)c * 32u, x);
            tc5::tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) x[i] = __float_as_uint(__uint_as_float(x[i]) * corr);
            tc5::tmem_st32(to + (uint32_t)c * 32u, x);
          }
          tc5::tmem_st_wait();
        }
        l *= corr;
        m = m_new;
      }
      if (!wait_warp(bar(B_PE + s), ph ^ 1u)) { ok = false; break; }
      const float m_use = (m == -INFINITY) ? 0.0f : m;
      float sum4[4] = {0.0f, 0.0f, 0.0f, 0.0f};
      const uint32_t prow = base + OFF_P + s * TILE_P + (uint32_t)row * 128u;
#pragma unroll
      for (int g = 0; g < 8; ++g) {    // 16-byte chunk g = columns 8g .. 8g+7
        float e[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          e[i] = ex2(fmaf(__uint_as_float(r[g >> 2][(g & 3) * 8 + i]), sl, -m_use));
          if (need_mask && col0 + g * 8 + i > lim) e[i] = 0.0f;
          sum4[i & 3] += e[i];
        }
        st_shared_v4(prow + ((((uint32_t)g) ^ swz) << 4), pack_bf16(e[0], e[1]), pack_bf16(e[2], e[3]), pack_bf16(e[4], e[5]),
                     pack_bf16(e[6], e[7]));
      }
      l += (sum4[0] + sum4[1]) + (sum4[2] + sum4[3]);
      tc5::fence_before_sync();
      fence_async_smem();
      __syncwarp();
      if (lane == 0) tc5::mbar_arrive(bar(B_PF + s));
    }
    ok = ok && wait_warp(bar(B_ACC), 0u);
    tc5::fence_after_sync();
    // merge the two groups: both halves of every row meet through shared memory (the Q tile is dead by now)
    float* xm = reinterpret_cast<float*>(smem + OFF_Q);    // [2][128] maxima, then [2][128] sums
    float* xl = xm + 256;
    xm[wg * 128 + row] = m;
    xl[wg * 128 + row] = l;
    asm volatile("bar.sync 1, 256;" ::: "memory");    // reached by all eight softmax warps, also after a failed wait
    if (ok) {
      const float m0 = xm[row], m1 = xm[128 + row], l0 = xl[row], l1 = xl[128 + row];
      const float mm = fmaxf(m0, m1);
      const float f0 = (m0 == -INFINITY) ? 0.0f : ex2(m0 - mm);
      const float f1 = (m1 == -INFINITY) ? 0.0f : ex2(m1 - mm);
      const float lt = l0 * f0 + l1 * f1;
      const float inv = lt > 0.0f ? 1.0f / lt : 0.0f;
      const float g0 = f0 * inv, g1 = f1 * inv;
      const bool two = n_kv > 1;    // with one key tile group 1 never wrote its accumulator
      __nv_bfloat16* dst = p.o + (int64_t)b * p.o_sb + (int64_t)grow * p.o_ss + (int64_t)h * p.o_sh + wg * 64;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t a0[32], a1[32];
        float v[32];
        tc5::tmem_ld32(tlane + TM_O + (uint32_t)wg * 64u + (uint32_t)c * 32u, a0);
        if (two) tc5::tmem_ld32(tlane + TM_O + 128u + (uint32_t)wg * 64u + (uint32_t)c * 32u, a1);
        tc5::tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(a0[i]) * g0;
        if (two) {
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = fmaf(__uint_as_float(a1[i]), g1, v[i]);
        }
        if (grow < p.seqlen) st_row32(dst + c * 32, v);
      }
      if (wg == 0 && grow < p.seqlen) p.lse[(int64_t)bh * p.seqlen + grow] = lt > 0.0f ? mm * kLn2 + logf(lt) : -INFINITY;
    }
  }

  // ---------------------------------------------------------------------- tear-down
  __syncwarp();
  if (*abort_flag) __nanosleep(200000);    // let copies / MMAs in flight finish before smem and TMEM go away
  tc5::fence_before_sync();
  __syncthreads();
  tc5::fence_after_sync();
  if (warp == 1) tc5::tmem_dealloc(tmem_base, TM_COLS);
}

// ====================================================================== forward, 128-key score tiles, P in tensor memory
namespace fwd2 {
constexpr int NK = 3;                         // ring depth of the K tiles (128 keys each)
constexpr int NV = 5;                         // ring depth of the V sub-tiles (64 keys each)
constexpr uint32_t PANEL_Q = 128 * 128;       // [128 query rows][64 bf16]
constexpr uint32_t TILE_Q = 2 * PANEL_Q;      // 32 KB
constexpr uint32_t PANEL_K = 128 * 128;       // [128 key rows][64 bf16]
constexpr uint32_t TILE_K = 2 * PANEL_K;      // 32 KB
constexpr uint32_t PANEL_V = 64 * 128;        // [64 key rows][64 bf16]
constexpr uint32_t TILE_V = 2 * PANEL_V;      // 16 KB
constexpr uint32_t OFF_Q = 0, OFF_K = TILE_Q, OFF_V = OFF_K + NK * TILE_K, OFF_X = OFF_V + NV * TILE_V, OFF_BAR = OFF_X + 2048;
enum { B_Q = 0, B_KF = 1, B_KE = B_KF + NK, B_VF = B_KE + NK, B_VE = B_VF + NV, B_SF = B_VE + NV, B_PF = B_SF + 2, B_OF = B_PF + 4,
       B_ACC = B_OF + 2, NBAR = B_ACC + 1 };
constexpr int SMEM = OFF_BAR + NBAR * 8 + 16 + 1024;
constexpr uint32_t TM_S = 0, TM_O = 256, TM_COLS = 512;    // two 128-column score slots, two 128-column outputs
constexpr float kRescaleStep = 8.0f;
}    // namespace fwd2

// Measured on this part: a 128 x N x 16 bf16 tcgen05.mma costs about 70 cycles for N = 64 as well as for N = 128 (the
// A operand, 4 KB, is fed at 64 B/clk whatever N is), wherever A comes from.  S = Q K^T is therefore issued over 128
// keys at a time (8 MMAs per 128 keys instead of 16).  The two softmax groups split every 128-key score tile by
// columns: group g owns keys [128 J + 64 g, 128 J + 64 g + 64) of tile J, with its own output accumulator O_g,
// reference maximum and row sum, exactly as if the groups took alternating 64-key tiles; the halves are merged once
// at the end.  Probabilities are packed to bf16 and stored with tcgen05.st over the first 32 columns of the 64-column
// half they were computed from, and O_g += P V reads them from tensor memory (no shared-memory round trip for P).
// The tensor pipe executes MMAs in issue order, so slot J & 1 may take the scores of tile J + 2 as soon as that MMA is
// issued after both PV products of tile J: no "slot free" barriers are needed.
__global__ void __launch_bounds__(kTcThreads, 1)
attn_fwd_tm_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                   const __grid_constant__ CUtensorMap map_v, const TcParams p) {
  using namespace fwd2;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = tc5::smem_u32(smem_raw);
  const uint32_t base = (raw_addr + 1023u) & ~1023u;
  uint8_t* smem = smem_raw + (base - raw_addr);
  const uint32_t bars = base + OFF_BAR;
  auto bar = [&](int i) { return bars + 8u * (uint32_t)i; };
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(smem + OFF_BAR + NBAR * 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);
  auto wait_warp = [&](uint32_t br, uint32_t ph) {
    return __all_sync(0xffffffffu, tc5::mbar_wait(br, ph, abort_flag, p.status, kStatusBit)) != 0;
  };

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int qt = (int)gridDim.x - 1 - (int)blockIdx.x;    // long rows first
  const int bh = blockIdx.y;
  const int b = bh / p.heads;
  const int h = bh - b * p.heads;
  const int q0 = qt * 128;
  const int n_all = (p.seqlen + 63) / 64;
  const int n_kv = p.causal ? min(2 * qt + 2, n_all) : n_all;    // 64-key sub-tiles with a visible key
  const int n_t = (n_kv + 1) >> 1;                               // 128-key tiles; a trailing odd sub-tile is fully masked

  if (threadIdx.x == 0) {
    tc5::mbar_init(bar(B_Q), 1);
    for (int s = 0; s < NK; ++s) {
      tc5::mbar_init(bar(B_KF + s), 1);
      tc5::mbar_init(bar(B_KE + s), 1);
    }
    for (int s = 0; s < NV; ++s) {
      tc5::mbar_init(bar(B_VF + s), 1);
      tc5::mbar_init(bar(B_VE + s), 1);
    }
    tc5::mbar_init(bar(B_SF + 0), 1);
    tc5::mbar_init(bar(B_SF + 1), 1);
    for (int s = 0; s < 4; ++s) tc5::mbar_init(bar(B_PF + s), 4);
    tc5::mbar_init(bar(B_OF + 0), 1);
    tc5::mbar_init(bar(B_OF + 1), 1);
    tc5::mbar_init(bar(B_ACC), 1);
    *abort_flag = 0;
    tc5::mbar_fence_init();
    tc5::tma_prefetch_desc(&map_q);
    tc5::tma_prefetch_desc(&map_k);
    tc5::tma_prefetch_desc(&map_v);
  }
  if (warp == 1) {
    tc5::tmem_alloc(tc5::smem_u32(tmem_holder), TM_COLS);
    tc5::tmem_relinquish();
  }
  tc5::fence_before_sync();
  __syncthreads();
  tc5::fence_after_sync();
  const uint32_t tmem_base = *tmem_holder;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      tc5::mbar_arrive_expect_tx(bar(B_Q), TILE_Q);
      tc5::tma_load_4d(base + OFF_Q, &map_q, 0, h, q0, b, bar(B_Q));
      tc5::tma_load_4d(base + OFF_Q + PANEL_Q, &map_q, 64, h, q0, b, bar(B_Q));
      bool ok = true;
      for (int t = 0; t < n_t && ok; ++t) {
        const int ks = t % NK;
        TC_WAIT(bar(B_KE + ks), ((uint32_t)(t / NK) & 1u) ^ 1u);
        tc5::mbar_arrive_expect_tx(bar(B_KF + ks), TILE_K);
        tc5::tma_load_4d(base + OFF_K + ks * TILE_K, &map_k, 0, h, t * 128, b, bar(B_KF + ks));
        tc5::tma_load_4d(base + OFF_K + ks * TILE_K + PANEL_K, &map_k, 64, h, t * 128, b, bar(B_KF + ks));
        for (int g = 0; g < 2; ++g) {
          const int j = 2 * t + g;
          const int vs = j % NV;
          if (!tc5::mbar_wait(bar(B_VE + vs), ((uint32_t)(j / NV) & 1u) ^ 1u, abort_flag, p.status, kStatusBit)) { ok = false; break; }
          tc5::mbar_arrive_expect_tx(bar(B_VF + vs), TILE_V);
          tc5::tma_load_4d(base + OFF_V + vs * TILE_V, &map_v, 0, h, j * 64, b, bar(B_VF + vs));
          tc5::tma_load_4d(base + OFF_V + vs * TILE_V + PANEL_V, &map_v, 64, h, j * 64, b, bar(B_VF + vs));
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (lane == 0) {
      const uint32_t idesc_s = tc5::idesc_bf16(128, 128, 0, 0);
      const uint32_t idesc_o = tc5::idesc_bf16(128, 128, 0, 1);
      // S[t & 1] = Q K_t^T over 128 keys
      auto issue_s = [&](int t) -> bool {
        const int ks = t % NK;
        if (!tc5::mbar_wait(bar(B_KF + ks), (uint32_t)(t / NK) & 1u, abort_flag, p.status, kStatusBit)) return false;
        tc5::fence_after_sync();
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
          const uint32_t off = (uint32_t)(kk >> 2) * PANEL_Q + (uint32_t)(kk & 3) * 32u;    // PANEL_K == PANEL_Q
          tc5::mma_f16(tmem_base + TM_S + (uint32_t)(t & 1) * 128u, tc5::smem_desc_k_sw128(base + OFF_Q + off),
                       tc5::smem_desc_k_sw128(base + OFF_K + ks * TILE_K + off), idesc_s, kk ? 1u : 0u);
        }
        tc5::mma_commit(bar(B_KE + ks));
        tc5::mma_commit(bar(B_SF + (t & 1)));
        return true;
      };
      do {
        TC_WAIT(bar(B_Q), 0u);
        bool ok = true;
        for (int t = 0; t < 2 && t < n_t; ++t)
          if (!issue_s(t)) { ok = false; break; }
        if (!ok) break;
        for (int t = 0; t < n_t && ok; ++t) {
          for (int g = 0; g < 2; ++g) {
            const int j = 2 * t + g;
            const int vs = j % NV;
            if (!tc5::mbar_wait(bar(B_PF + (t & 1) * 2 + g), (uint32_t)(t >> 1) & 1u, abort_flag, p.status, kStatusBit)) { ok = false; break; }
            if (!tc5::mbar_wait(bar(B_VF + vs), (uint32_t)(j / NV) & 1u, abort_flag, p.status, kStatusBit)) { ok = false; break; }
            tc5::fence_after_sync();
            // O_g (+)= P V : A = P from the first 32 columns of its half of the score slot, B = V with the key index as rows
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
              tc5::mma_f16_ta(tmem_base + TM_O + (uint32_t)g * 128u,
                              tmem_base + TM_S + (uint32_t)(t & 1) * 128u + (uint32_t)g * 64u + (uint32_t)kk * 8u,
                              tc5::smem_desc_mn_sw128(base + OFF_V + vs * TILE_V + (uint32_t)kk * 2048u, PANEL_V), idesc_o,
                              (t > 0 || kk) ? 1u : 0u);
            }
            tc5::mma_commit(bar(B_VE + vs));
            tc5::mma_commit(bar(B_OF + g));
          }
          if (ok && t + 2 < n_t && !issue_s(t + 2)) ok = false;
        }
        if (ok) tc5::mma_commit(bar(B_ACC));
      } while (false);
    }
  } else {
    // ------------------------------------------------------------------ softmax: one thread per query row and group
    const int qd = warp & 3;           // TMEM lane quarter this warp may access
    const int wg = (warp - 2) >> 2;    // group g: second index of the 64-key halves it owns
    const int row = qd * 32 + lane;
    const int grow = q0 + row;
    const uint32_t tlane = tmem_base + ((uint32_t)(qd * 32) << 16);
    const uint32_t to = tlane + TM_O + (uint32_t)wg * 128u;
    const float sl = p.scale * kLog2e;
    const int lim = p.causal ? min(grow, p.seqlen - 1) : p.seqlen - 1;    // last visible column
    float m = -INFINITY, l = 0.0f;    // reference maximum (log2 units) and row sum of this group
    bool ok = true;

    for (int t = 0; t < n_t; ++t) {
      const uint32_t ts = tlane + TM_S + (uint32_t)(t & 1) * 128u + (uint32_t)wg * 64u;
      if (!wait_warp(bar(B_SF + (t & 1)), (uint32_t)(t >> 1) & 1u)) { ok = false; break; }
      tc5::fence_after_sync();
      uint32_t r[2][32];
      tc5::tmem_ld32(ts, r[0]);
      tc5::tmem_ld32(ts + 32u, r[1]);
      tc5::tmem_ld_wait();
      const int col0 = (2 * t + wg) * 64;
      const bool need_mask = (p.causal && col0 + 63 > q0) || (col0 + 64 > p.seqlen);
      float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
      if (need_mask) {
#pragma unroll
        for (int i = 0; i < 64; ++i)
          if (col0 + i <= lim) mx4[i & 3] = fmaxf(mx4[i & 3], __uint_as_float(r[i >> 5][i & 31]));
      } else {
#pragma unroll
        for (int i = 0; i < 64; ++i) mx4[i & 3] = fmaxf(mx4[i & 3], __uint_as_float(r[i >> 5][i & 31]));
      }
      const float raw = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
      const float mx = raw == -INFINITY ? -INFINITY : raw * sl;    // no visible key: whatever the sign of the scale
      const bool grow_m = mx > m + kRescaleStep || (m == -INFINITY && mx > -INFINITY);
      if (__any_sync(0xffffffffu, grow_m)) {
        const float m_new = grow_m ? mx : m;
        const float corr = (m == -INFINITY) ? 0.0f : ex2(m - m_new);
        if (t > 0) {
          // every earlier product of this group must have landed in O before it is rescaled
          if (!wait_warp(bar(B_OF + wg), (uint32_t)(t - 1) & 1u)) { ok = false; break; }
          tc5::fence_after_sync();
#pragma unroll 1
          for (int c = 0; c < 4; ++c) {
            uint32_t x[32];
            tc5::tmem_ld32(to + (uint32_t)c * 32u, x);
            tc5::tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) x[i] = __float_as_uint(__uint_as_float(x[i]) * corr);
            tc5::tmem_st32(to + (uint32_t)c * 32u, x);
          }
        }
        l *= corr;
        m = m_new;
      }
      const float m_use = (m == -INFINITY) ? 0.0f : m;
      float sum4[4] = {0.0f, 0.0f, 0.0f, 0.0f};
      uint32_t pk[32];
#pragma unroll
      for (int g = 0; g < 8; ++g) {    // columns 8g .. 8g+7 -> packed columns 4g .. 4g+3
        float e[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          e[i] = ex2(fmaf(__uint_as_float(r[g >> 2][(g & 3) * 8 + i]), sl, -m_use));
          if (need_mask && col0 + g * 8 + i > lim) e[i] = 0.0f;
          sum4[i & 3] += e[i];
        }
        pk[4 * g] = pack_bf16(e[0], e[1]);
        pk[4 * g + 1] = pack_bf16(e[2], e[3]);
        pk[4 * g + 2] = pack_bf16(e[4], e[5]);
        pk[4 * g + 3] = pack_bf16(e[6], e[7]);
      }
      l += (sum4[0] + sum4[1]) + (sum4[2] + sum4[3]);
      tc5::tmem_st32(ts, pk);
      tc5::tmem_st_wait();    // also covers the rescaled accumulator
      tc5::fence_before_sync();
      __syncwarp();
      if (lane == 0) tc5::mbar_arrive(bar(B_PF + (t & 1) * 2 + wg));
    }
    ok = ok && wait_warp(bar(B_ACC), 0u);
    tc5::fence_after_sync();
    // merge the two groups: both halves of every row meet through shared memory
    float* xm = reinterpret_cast<float*>(smem + OFF_X);    // [2][128] maxima, then [2][128] sums
    float* xl = xm + 256;
    xm[wg * 128 + row] = m;
    xl[wg * 128 + row] = l;
    asm volatile("bar.sync 1, 256;" ::: "memory");    // reached by all eight softmax warps, also after a failed wait
    if (ok) {
      const float m0 = xm[row], m1 = xm[128 + row], l0 = xl[row], l1 = xl[128 + row];
      const float mm = fmaxf(m0, m1);
      const float f0 = (m0 == -INFINITY) ? 0.0f : ex2(m0 - mm);
      const float f1 = (m1 == -INFINITY) ? 0.0f : ex2(m1 - mm);
      const float lt = l0 * f0 + l1 * f1;
      const float inv = lt > 0.0f ? 1.0f / lt : 0.0f;
      const float g0 = f0 * inv, g1 = f1 * inv;
      // both accumulators were written (a group whose keys are all masked accumulated zeros)
      __nv_bfloat16* dst = p.o + (int64_t)b * p.o_sb + (int64_t)grow * p.o_ss + (int64_t)h * p.o_sh + wg * 64;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t a0[32], a1[32];
        float v[32];
        tc5::tmem_ld32(tlane + TM_O + (uint32_t)wg * 64u + (uint32_t)c * 32u, a0);
        tc5::tmem_ld32(tlane + TM_O + 128u + (uint32_t)wg * 64u + (uint32_t)c * 32u, a1);
        tc5::tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] = fmaf(__uint_as_float(a1[i]), g1, __uint_as_float(a0[i]) * g0);
        if (grow < p.seqlen) st_row32(dst + c * 32, v);
      }
      if (wg == 0 && grow < p.seqlen) p.lse[(int64_t)bh * p.seqlen + grow] = lt > 0.0f ? mm * kLn2 + logf(lt) : -INFINITY;
    }
  }

  // ---------------------------------------------------------------------- tear-down
  __syncwarp();
  if (*abort_flag) __nanosleep(200000);    // let copies / MMAs in flight finish before smem and TMEM go away
  tc5::fence_before_sync();
  __syncthreads();
  tc5::fence_after_sync();
  if (warp == 1) tc5::tmem_dealloc(tmem_base, TM_COLS);
}

// ============================================== forward, head size 128, many short rows: attn_fwd_tm_kernel over a list of items
namespace fwd2s {
using namespace fwd2;    // same tiles, rings and tensor-memory layout
constexpr uint32_t OFF_X3 = OFF_V + NV * TILE_V;          // two merge buffers of 2 KB (alternating work items)
constexpr uint32_t OFF_BAR3 = OFF_X3 + 4096;
enum { B3_QE = NBAR, B3_OE = NBAR + 1, B3_X = NBAR + 2, NBAR3 = NBAR + 3 };
constexpr int SMEM3 = OFF_BAR3 + NBAR3 * 8 + 16 + 1024;
}    // namespace fwd2s

// Work item -> (level, batch * head) for the persistent attention kernels: groups of G heads, inside a group by rising
// level (level 0 is the longest row), so that consecutive waves work on the same heads (their K / V or Q / dO stay in
// L2) and a walk that alternates direction per wave gives every CTA the same amount of work per group.
struct ItemOrder {
  int n_lv, bh_total, G;
  __device__ __forceinline__ void decode(int item, int& level, int& bh) const {
    const int g = item / (G * n_lv);
    const int hg = min(G, bh_total - g * G);
    const int j = item - g * G * n_lv;
    level = j / hg;
    bh = g * G + j % hg;
  }
};

// The schedule of attn_fwd_tm_kernel with one CTA per SM that walks the (query tile, batch * head) items.  Every ring (K, V, score
// slots) and every barrier keeps running across items, so the TMA warp loads Q, K and V of the next item while the softmax warps
// are still in the epilogue of the current one, and the MMA warp has the first two score tiles of the next item ready when they
// return.  B3_QE: all score MMAs of an item are complete, the Q tile may be overwritten; B3_OE: the softmax warps have read both
// accumulators, the first P V of the next item may overwrite them; B3_X: the eight softmax warps meet before the two groups'
// partial results are merged.  Bound by the exponentials and the groups' waits for each other (attn_fwd_ps_kernel has neither
// group wait, but one maximum per row instead of two: see the rule in msamp_attention_tc_fwd).
__global__ void __launch_bounds__(kTcThreads, 1)
attn_fwd_split_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                   const __grid_constant__ CUtensorMap map_v, const TcParams p, int n_qt, int n_items) {
  using namespace fwd2s;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = tc5::smem_u32(smem_raw);
  const uint32_t base = (raw_addr + 1023u) & ~1023u;
  uint8_t* smem = smem_raw + (base - raw_addr);
  const uint32_t bars = base + OFF_BAR3;
  auto bar = [&](int i) { return bars + 8u * (uint32_t)i; };
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(smem + OFF_BAR3 + NBAR3 * 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);
  auto wait_warp = [&](uint32_t br, uint32_t ph) {
    return __all_sync(0xffffffffu, tc5::mbar_wait(br, ph, abort_flag, p.status, kStatusBit)) != 0;
  };
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int n_all = (p.seqlen + 63) / 64;
  const ItemOrder order{n_qt, p.batch * p.heads, p.group};
  const int n_waves = (n_items + (int)gridDim.x - 1) / (int)gridDim.x;
  auto item_at = [&](int w) {
    const int c = (w & 1) ? (int)gridDim.x - 1 - (int)blockIdx.x : (int)blockIdx.x;
    return w * (int)gridDim.x + c;
  };
  auto item_tiles = [&](int qt) {
    const int n_kv = p.causal ? min(2 * qt + 2, n_all) : n_all;
    return (n_kv + 1) >> 1;
  };

  if (threadIdx.x == 0) {
    tc5::mbar_init(bar(B_Q), 1);
    for (int s = 0; s < NK; ++s) {
      tc5::mbar_init(bar(B_KF + s), 1);
      tc5::mbar_init(bar(B_KE + s), 1);
    }
    for (int s = 0; s < NV; ++s) {
      tc5::mbar_init(bar(B_VF + s), 1);
      tc5::mbar_init(bar(B_VE + s), 1);
    }
    tc5::mbar_init(bar(B_SF + 0), 1);
    tc5::mbar_init(bar(B_SF + 1), 1);
    for (int s = 0; s < 4; ++s) tc5::mbar_init(bar(B_PF + s), 4);
    tc5::mbar_init(bar(B_OF + 0), 1);
    tc5::mbar_init(bar(B_OF + 1), 1);
    tc5::mbar_init(bar(B_ACC), 1);
    tc5::mbar_init(bar(B3_QE), 1);
    tc5::mbar_init(bar(B3_OE), 8);
    tc5::mbar_init(bar(B3_X), 8);
    *abort_flag = 0;
    tc5::mbar_fence_init();
    tc5::tma_prefetch_desc(&map_q);
    tc5::tma_prefetch_desc(&map_k);
    tc5::tma_prefetch_desc(&map_v);
  }
  if (warp == 1) {
    tc5::tmem_alloc(tc5::smem_u32(tmem_holder), TM_COLS);
    tc5::tmem_relinquish();
  }
  tc5::fence_before_sync();
  __syncthreads();
  tc5::fence_after_sync();
  const uint32_t tmem_base = *tmem_holder;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      int gt = 0;    // 128-key tiles loaded so far (all items)
      bool ok = true;
      int it = 0;
      for (int w = 0; w < n_waves && ok; ++w) {
        const int item = item_at(w);
        if (item >= n_items) continue;
        int level, bh;
        order.decode(item, level, bh);
        const int qt = n_qt - 1 - level;
        const int b = bh / p.heads, h = bh - b * p.heads;
        const int n_t = item_tiles(qt);
        if (it > 0 && !tc5::mbar_wait(bar(B3_QE), (uint32_t)(it - 1) & 1u, abort_flag, p.status, kStatusBit)) break;
        tc5::mbar_arrive_expect_tx(bar(B_Q), TILE_Q);
        tc5::tma_load_4d(base + OFF_Q, &map_q, 0, h, qt * 128, b, bar(B_Q));
        tc5::tma_load_4d(base + OFF_Q + PANEL_Q, &map_q, 64, h, qt * 128, b, bar(B_Q));
        for (int t = 0; t < n_t && ok; ++t, ++gt) {
          const int ks = gt % NK;
          if (!tc5::mbar_wait(bar(B_KE + ks), ((uint32_t)(gt / NK) & 1u) ^ 1u, abort_flag, p.status, kStatusBit)) { ok = false; break; }
          tc5::mbar_arrive_expect_tx(bar(B_KF + ks), TILE_K);
          tc5::tma_load_4d(base + OFF_K + ks * TILE_K, &map_k, 0, h, t * 128, b, bar(B_KF + ks));
          tc5::tma_load_4d(base + OFF_K + ks * TILE_K + PANEL_K, &map_k, 64, h, t * 128, b, bar(B_KF + ks));
          for (int g = 0; g < 2; ++g) {
            const int gj = 2 * gt + g;    // 64-key sub-tiles loaded so far
            const int vs = gj % NV;
            if (!tc5::mbar_wait(bar(B_VE + vs), ((uint32_t)(gj / NV) & 1u) ^ 1u, abort_flag, p.status, kStatusBit)) { ok = false; break; }
            tc5::mbar_arrive_expect_tx(bar(B_VF + vs), TILE_V);
            tc5::tma_load_4d(base + OFF_V + vs * TILE_V, &map_v, 0, h, (2 * t + g) * 64, b, bar(B_VF + vs));
            tc5::tma_load_4d(base + OFF_V + vs * TILE_V + PANEL_V, &map_v, 64, h, (2 * t + g) * 64, b, bar(B_VF + vs));
          }
        }
        ++it;
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (lane == 0) {
      const uint32_t idesc_s = tc5::idesc_bf16(128, 128, 0, 0);
      const uint32_t idesc_o = tc5::idesc_bf16(128, 128, 0, 1);
      auto issue_s = [&](int gs) -> bool {    // S[gs & 1] = Q K^T for the gs-th tile of this CTA
        const int ks = gs % NK;
        if (!tc5::mbar_wait(bar(B_KF + ks), (uint32_t)(gs / NK) & 1u, abort_flag, p.status, kStatusBit)) return false;
        tc5::fence_after_sync();
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
          const uint32_t off = (uint32_t)(kk >> 2) * PANEL_Q + (uint32_t)(kk & 3) * 32u;
          tc5::mma_f16(tmem_base + TM_S + (uint32_t)(gs & 1) * 128u, tc5::smem_desc_k_sw128(base + OFF_Q + off),
                       tc5::smem_desc_k_sw128(base + OFF_K + ks * TILE_K + off), idesc_s, kk ? 1u : 0u);
        }
        tc5::mma_commit(bar(B_KE + ks));
        tc5::mma_commit(bar(B_SF + (gs & 1)));
        return true;
      };
      int g0 = 0;    // tiles of earlier items
      bool ok = true;
      int it = 0;
      for (int w = 0; w < n_waves && ok; ++w) {
        const int item = item_at(w);
        if (item >= n_items) continue;
        int level, bh;
        order.decode(item, level, bh);
        const int n_t = item_tiles(n_qt - 1 - level);
        if (!tc5::mbar_wait(bar(B_Q), (uint32_t)it & 1u, abort_flag, p.status, kStatusBit)) { ok = false; break; }
        for (int t = 0; t < 2 && t < n_t; ++t)
          if (!issue_s(g0 + t)) { ok = false; break; }
        if (!ok) break;
        if (n_t <= 2) tc5::mma_commit(bar(B3_QE));    // every score product of this item has been issued
        // the softmax warps must have read the previous item's accumulators before they are overwritten
        if (it > 0 && !tc5::mbar_wait(bar(B3_OE), (uint32_t)(it - 1) & 1u, abort_flag, p.status, kStatusBit)) { ok = false; break; }
        for (int t = 0; t < n_t && ok; ++t) {
          const int gs = g0 + t;
          for (int g = 0; g < 2; ++g) {
            const int gj = 2 * gs + g;
            const int vs = gj % NV;
            // the data barrier first: a wait costs 100+ cycles even when its phase completed long ago, and this one
            // then passes while the softmax warps are still at work on P
            if (!tc5::mbar_wait(bar(B_VF + vs), (uint32_t)(gj / NV) & 1u, abort_flag, p.status, kStatusBit)) { ok = false; break; }
            if (!tc5::mbar_wait(bar(B_PF + (gs & 1) * 2 + g), (uint32_t)(gs >> 1) & 1u, abort_flag, p.status, kStatusBit)) { ok = false; break; }
            tc5::fence_after_sync();
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
              tc5::mma_f16_ta(tmem_base + TM_O + (uint32_t)g * 128u,
                              tmem_base + TM_S + (uint32_t)(gs & 1) * 128u + (uint32_t)g * 64u + (uint32_t)kk * 8u,
                              tc5::smem_desc_mn_sw128(base + OFF_V + vs * TILE_V + (uint32_t)kk * 2048u, PANEL_V), idesc_o,
                              (t > 0 || kk) ? 1u : 0u);
            }
            tc5::mma_commit(bar(B_VE + vs));
            tc5::mma_commit(bar(B_OF + g));
          }
          if (ok && t + 2 < n_t) {
            if (!issue_s(gs + 2)) { ok = false; break; }
            if (t + 3 == n_t) tc5::mma_commit(bar(B3_QE));
          }
        }
        if (ok) tc5::mma_commit(bar(B_ACC));
        g0 += n_t;
        ++it;
      }
    }
  } else {
    // ------------------------------------------------------------------ softmax: one thread per query row and group
    const int qd = warp & 3;           // TMEM lane quarter this warp may access
    const int wg = (warp - 2) >> 2;    // group g: second index of the 64-key halves it owns
    const int row = qd * 32 + lane;
    const uint32_t tlane = tmem_base + ((uint32_t)(qd * 32) << 16);
    const uint32_t to = tlane + TM_O + (uint32_t)wg * 128u;
    const float sl = p.scale * kLog2e;
    int g0 = 0;
    bool ok = true;
    int it = 0;
    for (int w = 0; w < n_waves; ++w) {
      const int item = item_at(w);
      if (item >= n_items) continue;
      int level, bh;
      order.decode(item, level, bh);
      const int qt = n_qt - 1 - level;
      const int b = bh / p.heads, h = bh - b * p.heads;
      const int n_t = item_tiles(qt);
      const int q0 = qt * 128;
      const int grow = q0 + row;
      const int lim = p.causal ? min(grow, p.seqlen - 1) : p.seqlen - 1;    // last visible column
      float m = -INFINITY, l = 0.0f;    // reference maximum (log2 units) and row sum of this group
      for (int t = 0; t < n_t; ++t) {
        const int gs = g0 + t;
        const uint32_t ts = tlane + TM_S + (uint32_t)(gs & 1) * 128u + (uint32_t)wg * 64u;
        if (!wait_warp(bar(B_SF + (gs & 1)), (uint32_t)(gs >> 1) & 1u)) { ok = false; break; }
        tc5::fence_after_sync();
        uint32_t r[2][32];
        tc5::tmem_ld32(ts, r[0]);
        tc5::tmem_ld32(ts + 32u, r[1]);
        tc5::tmem_ld_wait();
        const int col0 = (2 * t + wg) * 64;
        const bool need_mask = (p.causal && col0 + 63 > q0) || (col0 + 64 > p.seqlen);
        float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
        if (need_mask) {
#pragma unroll
          for (int i = 0; i < 64; ++i)
            if (col0 + i <= lim) mx4[i & 3] = fmaxf(mx4[i & 3], __uint_as_float(r[i >> 5][i & 31]));
        } else {
#pragma unroll
          for (int i = 0; i < 64; ++i) mx4[i & 3] = fmaxf(mx4[i & 3], __uint_as_float(r[i >> 5][i & 31]));
        }
        const float raw = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
        const float mx = raw == -INFINITY ? -INFINITY : raw * sl;
        const bool grow_m = mx > m + kRescaleStep || (m == -INFINITY && mx > -INFINITY);
        if (__any_sync(0xffffffffu, grow_m)) {
          const float m_new = grow_m ? mx : m;
          const float corr = (m == -INFINITY) ? 0.0f : ex2(m - m_new);
          if (t > 0) {
            // every earlier product of this group and item must have landed in O before it is rescaled
            if (!wait_warp(bar(B_OF + wg), (uint32_t)(gs - 1) & 1u)) { ok = false; break; }
            tc5::fence_after_sync();
#pragma unroll 1
            for (int c = 0; c < 4; ++c) {
              uint32_t x[32];
              tc5::tmem_ld32(to + (uint32_t)c * 32u, x);
              tc5::tmem_ld_wait();
#pragma unroll
              for (int i = 0; i < 32; ++i) x[i] = __float_as_uint(__uint_as_float(x[i]) * corr);
              tc5::tmem_st32(to + (uint32_t)c * 32u, x);
            }
          }
          l *= corr;
          m = m_new;
        }
        const float m_use = (m == -INFINITY) ? 0.0f : m;
        float sum4[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        uint32_t pk[32];
#pragma unroll
        for (int g = 0; g < 8; ++g) {    // columns 8g .. 8g+7 -> packed columns 4g .. 4g+3
          float e[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            e[i] = ex2(fmaf(__uint_as_float(r[g >> 2][(g & 3) * 8 + i]), sl, -m_use));
            if (need_mask && col0 + g * 8 + i > lim) e[i] = 0.0f;
            sum4[i & 3] += e[i];
          }
          pk[4 * g] = pack_bf16(e[0], e[1]);
          pk[4 * g + 1] = pack_bf16(e[2], e[3]);
          pk[4 * g + 2] = pack_bf16(e[4], e[5]);
          pk[4 * g + 3] = pack_bf16(e[6], e[7]);
        }
        l += (sum4[0] + sum4[1]) + (sum4[2] + sum4[3]);
        tc5::tmem_st32(ts, pk);
        tc5::tmem_st_wait();    // also covers the rescaled accumulator
        tc5::fence_before_sync();
        __syncwarp();
        if (lane == 0) tc5::mbar_arrive(bar(B_PF + (gs & 1) * 2 + wg));
      }
      ok = ok && wait_warp(bar(B_ACC), (uint32_t)it & 1u);
      tc5::fence_after_sync();
      // merge the two groups through shared memory (two buffers, alternating items: a warp that is already in the next
      // item's merge cannot overwrite values another warp still reads)
      float* xm = reinterpret_cast<float*>(smem + OFF_X3 + (uint32_t)(it & 1) * 2048u);    // [2][128] maxima, then [2][128] sums
      float* xl = xm + 256;
      if (!ok) break;
      xm[wg * 128 + row] = m;
      xl[wg * 128 + row] = l;
      // the eight warps meet on an mbarrier (bounded wait) rather than on a named barrier: a warp that gave up on an
      // earlier wait leaves without arriving, and the others then give up here instead of waiting for it for ever
      __syncwarp();
      if (lane == 0) tc5::mbar_arrive(bar(B3_X));
      if (!wait_warp(bar(B3_X), (uint32_t)it & 1u)) { ok = false; break; }
      const float m0 = xm[row], m1 = xm[128 + row], l0 = xl[row], l1 = xl[128 + row];
      const float mm = fmaxf(m0, m1);
      const float f0 = (m0 == -INFINITY) ? 0.0f : ex2(m0 - mm);
      const float f1 = (m1 == -INFINITY) ? 0.0f : ex2(m1 - mm);
      const float lt = l0 * f0 + l1 * f1;
      const float inv = lt > 0.0f ? 1.0f / lt : 0.0f;
      const float gg0 = f0 * inv, gg1 = f1 * inv;
      uint32_t a0[2][32], a1[2][32];
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        tc5::tmem_ld32(tlane + TM_O + (uint32_t)wg * 64u + (uint32_t)c * 32u, a0[c]);
        tc5::tmem_ld32(tlane + TM_O + 128u + (uint32_t)wg * 64u + (uint32_t)c * 32u, a1[c]);
      }
      tc5::tmem_ld_wait();
      tc5::fence_before_sync();
      __syncwarp();
      if (lane == 0) tc5::mbar_arrive(bar(B3_OE));    // the accumulators may take the next item
      __nv_bfloat16* dst = p.o + (int64_t)b * p.o_sb + (int64_t)grow * p.o_ss + (int64_t)h * p.o_sh + wg * 64;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        float v[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] = fmaf(__uint_as_float(a1[c][i]), gg1, __uint_as_float(a0[c][i]) * gg0);
        if (grow < p.seqlen) st_row32(dst + c * 32, v);
      }
      if (wg == 0 && grow < p.seqlen) p.lse[(int64_t)bh * p.seqlen + grow] = lt > 0.0f ? mm * kLn2 + logf(lt) : -INFINITY;
      g0 += n_t;
      ++it;
    }
  }

  // ---------------------------------------------------------------------- tear-down
  __syncwarp();
  if (*abort_flag) __nanosleep(200000);    // let copies / MMAs in flight finish before smem and TMEM go away
  tc5::fence_before_sync();
  __syncthreads();
  tc5::fence_after_sync();
  if (warp == 1) tc5::tmem_dealloc(tmem_base, TM_COLS);
}

// ================================================================= forward, persistent CTAs over (query tile, batch, head)
// Thread layout of the persistent kernels: one warpgroup of which warp 0 issues TMA and warp 1 the MMAs, and two warpgroups
// of softmax threads.  The register file is split by setmaxnreg: AUX for the first, (384 * 168 - 128 * AUX) / 256 for the
// other two, which adds up to what the launch holds (384 threads x 168).
constexpr int kPsThreads = 384;
constexpr int softmax_regs(int aux) { return (384 * 168 - 128 * aux) / 256; }
template <int AUX>
__device__ __forceinline__ void regs_aux() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(AUX)); }
template <int AUX>
__device__ __forceinline__ void regs_softmax() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(softmax_regs(AUX))); }

// Position in a ring of N slots and the parity of its current round.
template <int N>
struct Ring {
  int slot = 0;
  uint32_t phase = 0;
  __device__ __forceinline__ void next() {
    if (++slot == N) {
      slot = 0;
      phase ^= 1u;
    }
  }
};

namespace fwd3 {
constexpr uint32_t PANEL = 128 * 128;    // [128 rows][64 bf16]: one 64-wide slice of the head
template <int D>
struct Cfg {
  static constexpr int HP = D / 64;
  static constexpr int NA = D == 128 ? 1 : 2;    // running maxima, row sums and accumulators of a row, one per 128 / NA columns of a tile
  static constexpr int NK = D == 128 ? 3 : 4, NV = D == 128 ? 2 : 4;    // ring depths of the K and V tiles (128 keys each)
  static constexpr uint32_t TILE = HP * PANEL;
  static constexpr uint32_t OFF_K = 2 * TILE, OFF_V = OFF_K + NK * TILE, OFF_BAR = OFF_V + NV * TILE;    // two Q tiles first
  static constexpr int B_Q = 0, B_QE = 2, B_KF = 4, B_KE = B_KF + NK, B_VF = B_KE + NK, B_VE = B_VF + NV, B_SF = B_VE + NV, B_SE = B_SF + 2,
                       B_PF = B_SE + 1, B_OF = B_PF + 2, B_X = B_OF + 2, NBAR = B_X + 1;
  static constexpr int SMEM = OFF_BAR + NBAR * 8 + 16 + 1024;
  static_assert(SMEM <= 227 * 1024, "persistent forward kernel: shared memory");
};
// scores (128 columns), P of each group (64), accumulators of each group (NA * D = 128)
constexpr int kFwdAux = 72;    // registers of the TMA and MMA threads
constexpr uint32_t TM_S = 0, TM_P = 128, TM_O = 256, TM_COLS = 512;
constexpr int kExactTiles = 4;          // head size 128: the maximum is exact for the first tiles of a row, then it may
constexpr float kRescaleStep = 4.0f;    // lag the true one by 2^4
}    // namespace fwd3

// Work item (query tile, batch * head) lists of the forward kernel.  Stream g of CTA c is worker g * CTAs + c and takes one
// item per wave of 2 * CTAs items.  When what is left for the last wave is no more than one item per CTA, the two streams
// of a CTA share its item (stream g takes key tiles g, g + 2, ...) and merge their halves at the end: a stream by itself
// needs 1.7 times as long per tile as two streams together.
struct FwdItem {
  int qt, bh;
  int first, step, n_t;    // key tiles first, first + step, ... < n_t; n_t == 0: no item
  bool shared;
};
struct FwdItems {
  int n_qt, n_items, bh_total, G, n_ctas, causal;
  __device__ __forceinline__ FwdItem at(int w, int g) const {
    const int full = n_items / (2 * n_ctas), rem = n_items - full * 2 * n_ctas;
    const int c = (int)blockIdx.x;
    FwdItem x{0, 0, 0, 1, 0, false};
    // even waves upwards, odd waves downwards, so that the sums per worker stay within about a tile of each other
    int j = g * n_ctas + c;
    if (w & 1) j = 2 * n_ctas - 1 - j;
    if (w >= full) {
      if (w > full) return x;
      x.shared = rem <= n_ctas;
      if (x.shared) {
        j = c;
        x.first = g;
        x.step = 2;
      } else {
        j = g * n_ctas + c;
      }
      if (j >= rem) return x;
    }
    // Items are ordered in groups of G (batch, head) pairs, inside a group by falling query tile (= falling length), so
    // that the CTAs of a few consecutive waves work on the same heads: a head's K and V are read from HBM by its longest
    // rows and found in L2 by the others (with all heads of one query-tile level in a wave the kernel read K / V 3.9 times).
    const int item = w * 2 * n_ctas + j;
    const int grp = item / (G * n_qt);
    const int hg = min(G, bh_total - grp * G);
    const int k = item - grp * G * n_qt;
    x.qt = n_qt - 1 - k / hg;
    x.bh = grp * G + k % hg;
    x.n_t = causal ? x.qt + 1 : n_qt;
    return x;
  }
};

// The tiles of a CTA in the order in which the tensor pipe takes them: the two streams in turn, one tile each, until both
// lists are exhausted.  The TMA thread and the two MMA threads walk the same sequence.
struct FwdStream {
  int g, w, t;           // stream, next wave, tile of the current item
  FwdItem item;          // n_t == 0: list exhausted
  uint32_t started;      // items so far (an item that is one shared tile leaves the second stream without any)
  __device__ __forceinline__ void open(const FwdItems& items) {
    item = items.at(w++, g);
    t = item.first;
    if (t >= item.n_t) item.n_t = 0;
    else ++started;
  }
  __device__ __forceinline__ bool first() const { return t == item.first; }
  __device__ __forceinline__ bool last() const { return t + item.step >= item.n_t; }
};
struct FwdSeq {
  FwdStream cur, other;
  __device__ __forceinline__ FwdSeq(const FwdItems& items) {
    cur.g = cur.w = other.w = 0;
    other.g = 1;
    cur.started = other.started = 0u;
    cur.open(items);    // stream 0 has an item in every CTA
    other.open(items);
  }
  __device__ __forceinline__ bool more() const { return cur.item.n_t > 0; }
  __device__ __forceinline__ void advance(const FwdItems& items) {
    cur.t += cur.item.step;
    if (cur.t >= cur.item.n_t) cur.open(items);
    if (other.item.n_t > 0) {
      const FwdStream x = cur;
      cur = other;
      other = x;
    }
  }
};

// One CTA per SM; its two softmax groups (one thread per query row) each walk their own list of work items (query tile,
// batch * head) against key tiles of 128, and never exchange anything.  The tensor pipe serves the two streams in turn.
// What bounds it, per tile of 128 x 128: 1024 cycles of MUFU (16384 exponentials at 16 a clock), 12 to 16 MMAs of about 70
// cycles (a 128 x N x 16 bf16 MMA costs that for N = 64 and for N = 128: the 4 KB A operand is fed at 64 B/clk), and some
// 1200 cycles of maxima, sums, packing and TMEM traffic of one group, which only the other group's exponentials hide.
//  * P is relative to the row's running maximum, so that the largest probability is exactly 1 and rounds to bf16 without error: with a
//    reference that lagged by up to 2^8 the output of peaked rows was up to 20 % further from 64 bits (scores of standard deviation
//    2, 2048 keys of 64).  Head size 64 has tensor memory for two accumulators per row and takes a maximum per 64 keys, as a 64-key
//    tile would: never further off than the mma.sync kernels (64 x 197 rows: 0.00212 against 0.00215).  Head size 128 has one, exact
//    over the first kExactTiles tiles of a row; later the weights are spread, and a lag of 2^4 saves most rescales (2 % of the time
//    at 2048 and 4096 rows).  The exact maximum costs 7 % of the time at 64 (8 x 1024 x 12 heads, causal: 41 -> 43.5 us) and 3 % at
//    128; a rescale moves all columns through registers at once.
//  * A group reads its 128 scores into registers and releases the one score slot at once, so that the scores of the next
//    tile (the other group's) are there before they are needed; P goes to a place of its own, from where O_g += P V reads
//    it as a TMEM operand.  When P was written over the scores, a group waited 1500 of 3950 cycles per tile for its next
//    scores, which had to wait for the product that read P.
//  * Streams of whole items keep the groups out of phase, and one group's epilogue runs under the other's tiles; two groups
//    that split every tile, or alternated on the tiles of one item, met at the MUFU and at every item's end.
//  * The tensor pipe buffers next to nothing and a wait or a commit costs the issuing thread 50 to 250 cycles, so one thread
//    that issued both products kept the pipe idle for half of the tile.  Two threads of two warps issue them; nothing
//    depends on the order between the two, every reuse below is a barrier.  Both probe their next tile while MMAs run.
// Measured, forward only, against one stream of tiles that both groups split: 4 x 2048 x 32 heads of 128, causal, 204 -> 190 to
// 194 us; 2 x 4096 x 16 heads of 128, causal, 242 -> 208 us; 1 x 8192 x 16, 433 -> 328 us.
// Reuse: Q_g after the last score product of its item (B_QE); the score slot after B_SE (tiles in sequence order); P_g and
// the accumulator after P V of the group's previous tile (B_OF); the accumulator of a finished item is read before the group
// hands over its next P (B_PF), so the next item's first product cannot overtake it.
template <int D>
__global__ void __launch_bounds__(kPsThreads, 1)
attn_fwd_ps_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                   const __grid_constant__ CUtensorMap map_v, const TcParams p, int n_qt, int n_items) {
  using namespace fwd3;
  using C = Cfg<D>;
  constexpr int HP = C::HP, NK = C::NK, NV = C::NV, NA = C::NA;
  constexpr uint32_t TILE = C::TILE, OFF_Q = 0, OFF_K = C::OFF_K, OFF_V = C::OFF_V;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = tc5::smem_u32(smem_raw);
  const uint32_t base = (raw_addr + 1023u) & ~1023u;
  uint8_t* smem = smem_raw + (base - raw_addr);
  const uint32_t bars = base + C::OFF_BAR;
  auto bar = [&](int i) { return bars + 8u * (uint32_t)i; };
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(smem + C::OFF_BAR + C::NBAR * 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);
  auto wait = [&](uint32_t br, uint32_t ph) { return tc5::mbar_wait(br, ph, abort_flag, p.status, kStatusBit); };
  auto wait_warp = [&](uint32_t br, uint32_t ph) { return __all_sync(0xffffffffu, wait(br, ph)) != 0; };
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const FwdItems items{n_qt, n_items, p.batch * p.heads, p.group, (int)gridDim.x, p.causal};

  if (threadIdx.x == 0) {
    for (int g = 0; g < 2; ++g) {
      tc5::mbar_init(bar(C::B_Q + g), 1);
      tc5::mbar_init(bar(C::B_QE + g), 1);
      tc5::mbar_init(bar(C::B_SF + g), 1);
      tc5::mbar_init(bar(C::B_PF + g), 4);
      tc5::mbar_init(bar(C::B_OF + g), 1);
    }
    tc5::mbar_init(bar(C::B_SE), 4);
    tc5::mbar_init(bar(C::B_X), 8);
    for (int s = 0; s < NK; ++s) {
      tc5::mbar_init(bar(C::B_KF + s), 1);
      tc5::mbar_init(bar(C::B_KE + s), 1);
    }
    for (int s = 0; s < NV; ++s) {
      tc5::mbar_init(bar(C::B_VF + s), 1);
      tc5::mbar_init(bar(C::B_VE + s), 1);
    }
    *abort_flag = 0;
    tc5::mbar_fence_init();
    tc5::tma_prefetch_desc(&map_q);
    tc5::tma_prefetch_desc(&map_k);
    tc5::tma_prefetch_desc(&map_v);
  }
  if (warp == 1) {
    tc5::tmem_alloc(tc5::smem_u32(tmem_holder), TM_COLS);
    tc5::tmem_relinquish();
  }
  tc5::fence_before_sync();
  __syncthreads();
  tc5::fence_after_sync();
  const uint32_t tmem_base = *tmem_holder;

  if (warp < 4) {
    regs_aux<kFwdAux>();
    if (warp == 0 && lane == 0) {
      // ---------------------------------------------------------------- TMA producer
      FwdSeq seq(items);
      Ring<NK> kr;
      Ring<NV> vr;
      // K runs two tiles ahead of V, as the score products run ahead of P V: a V tile waits for the product of an earlier one
      int vt0 = 0, vbh0 = 0, vt1 = 0, vbh1 = 0, waiting = 0;
      while (seq.more() || waiting > 0) {
        const bool more = seq.more();
        const int g = seq.cur.g, t = seq.cur.t, bh = seq.cur.item.bh;
        if (more) {
          const int b = bh / p.heads, h = bh - b * p.heads;
          if (seq.cur.first()) {
            if (seq.cur.started > 1 && !wait(bar(C::B_QE + g), seq.cur.started & 1u)) break;    // the previous item's phase
            tc5::mbar_arrive_expect_tx(bar(C::B_Q + g), TILE);
#pragma unroll
            for (int pp = 0; pp < HP; ++pp)
              tc5::tma_load_4d(base + OFF_Q + g * TILE + pp * PANEL, &map_q, pp * 64, h, seq.cur.item.qt * 128, b, bar(C::B_Q + g));
          }
          if (!wait(bar(C::B_KE + kr.slot), kr.phase ^ 1u)) break;
          tc5::mbar_arrive_expect_tx(bar(C::B_KF + kr.slot), TILE);
#pragma unroll
          for (int pp = 0; pp < HP; ++pp)
            tc5::tma_load_4d(base + OFF_K + kr.slot * TILE + pp * PANEL, &map_k, pp * 64, h, t * 128, b, bar(C::B_KF + kr.slot));
          kr.next();
        }
        if (waiting == 2 || !more) {
          const int b = vbh0 / p.heads, h = vbh0 - b * p.heads;
          if (!wait(bar(C::B_VE + vr.slot), vr.phase ^ 1u)) break;
          tc5::mbar_arrive_expect_tx(bar(C::B_VF + vr.slot), TILE);
#pragma unroll
          for (int pp = 0; pp < HP; ++pp)
            tc5::tma_load_4d(base + OFF_V + vr.slot * TILE + pp * PANEL, &map_v, pp * 64, h, vt0 * 128, b, bar(C::B_VF + vr.slot));
          vr.next();
          vt0 = vt1;
          vbh0 = vbh1;
          --waiting;
        }
        if (more) {
          (waiting == 0 ? vt0 : vt1) = t;
          (waiting == 0 ? vbh0 : vbh1) = bh;
          ++waiting;
          seq.advance(items);
        }
      }
    } else if (warp == 1 && lane == 0) {
      // ---------------------------------------------------------------- S = Q K^T, tile by tile of the sequence
      const uint32_t idesc = tc5::idesc_bf16(128, 128, 0, 0);
      FwdSeq seq(items);
      Ring<NK> kr;
      bool k_ready = false;    // probe of the next K tile, made while the MMAs of this one run
      for (uint32_t n = 0; seq.more(); ++n) {
        const int g = seq.cur.g;
        if (seq.cur.first() && !wait(bar(C::B_Q + g), (seq.cur.started - 1) & 1u)) break;
        if (!k_ready && !wait(bar(C::B_KF + kr.slot), kr.phase)) break;
        if (n > 0 && !wait(bar(C::B_SE), (n - 1) & 1u)) break;    // the previous scores have been read
        tc5::fence_after_sync();
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          const uint32_t off = (uint32_t)(kk >> 2) * PANEL + (uint32_t)(kk & 3) * 32u;
          tc5::mma_f16(tmem_base + TM_S, tc5::smem_desc_k_sw128(base + OFF_Q + g * TILE + off),
                       tc5::smem_desc_k_sw128(base + OFF_K + kr.slot * TILE + off), idesc, kk ? 1u : 0u);
        }
        tc5::mma_commit(bar(C::B_SF + g));
        tc5::mma_commit(bar(C::B_KE + kr.slot));
        if (seq.cur.last()) tc5::mma_commit(bar(C::B_QE + g));    // last score product of the item
        kr.next();
        k_ready = tc5::mbar_test(bar(C::B_KF + kr.slot), kr.phase);
        seq.advance(items);
      }
    } else if (warp == 2 && lane == 0) {
      // ---------------------------------------------------------------- O_g += P V, in the same order
      const uint32_t idesc = tc5::idesc_bf16(128, D, 0, 1);
      FwdSeq seq(items);
      Ring<NV> vr;
      bool v_ready = false;
      uint32_t p_phase = 0u;    // bit g: parity of stream g's next P
      for (; seq.more(); seq.advance(items)) {
        const int g = seq.cur.g;
        const bool first = seq.cur.first();
        if (!v_ready && !wait(bar(C::B_VF + vr.slot), vr.phase)) break;
        if (!wait(bar(C::B_PF + g), (p_phase >> g) & 1u)) break;
        p_phase ^= 1u << g;
        tc5::fence_after_sync();
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
          const int a = kk / (8 / NA);    // accumulator of these 16 keys
          tc5::mma_f16_ta(tmem_base + TM_O + (uint32_t)(g * 128 + a * D), tmem_base + TM_P + (uint32_t)g * 64u + (uint32_t)kk * 8u,
                          tc5::smem_desc_mn_sw128(base + OFF_V + vr.slot * TILE + (uint32_t)kk * 2048u, PANEL), idesc,
                          (!first || kk % (8 / NA)) ? 1u : 0u);
        }
        tc5::mma_commit(bar(C::B_OF + g));
        tc5::mma_commit(bar(C::B_VE + vr.slot));
        vr.next();
        v_ready = tc5::mbar_test(bar(C::B_VF + vr.slot), vr.phase);
      }
    }
  } else {
    regs_softmax<kFwdAux>();
    // ------------------------------------------------------------------ softmax: one thread per query row
    const int qd = warp & 3;           // TMEM lane quarter this warp may access
    const int wg = (warp - 4) >> 2;    // stream
    const int row = qd * 32 + lane;
    const uint32_t tlane = tmem_base + ((uint32_t)(qd * 32) << 16);
    const uint32_t ts = tlane + TM_S, tp = tlane + TM_P + (uint32_t)wg * 64u, to = tlane + TM_O + (uint32_t)wg * 128u;
    const float sl = p.scale * kLog2e;
    const uint64_t sl2 = f2_pack(sl, sl);
    uint32_t n = 0;    // tiles of this stream so far
    bool ok = true;
    for (int w = 0; ok; ++w) {
      const FwdItem item = items.at(w, wg);
      if (item.n_t == 0) break;
      const int qt = item.qt, bh = item.bh, n_t = item.n_t;
      const int b = bh / p.heads, h = bh - b * p.heads;
      const int q0 = qt * 128;
      const int grow = q0 + row;
      const int lim = p.causal ? min(grow, p.seqlen - 1) : p.seqlen - 1;    // last visible column
      const int wlim = p.causal ? min(q0 + qd * 32 + 31, p.seqlen - 1) : p.seqlen - 1;    // the same for the warp's last row
      float m[NA], l[NA];    // running maximum (log2 units) and row sum
#pragma unroll
      for (int a = 0; a < NA; ++a) {
        m[a] = -INFINITY;
        l[a] = 0.0f;
      }
      for (int t = item.first; t < n_t; t += item.step, ++n) {
        if (!wait_warp(bar(C::B_SF + wg), n & 1u)) { ok = false; break; }
        tc5::fence_after_sync();
        uint32_t r[4][32];
#pragma unroll
        for (int c = 0; c < 4; ++c) tc5::tmem_ld32(ts + 32u * c, r[c]);
        tc5::tmem_ld_wait();
        tc5::fence_before_sync();
        __syncwarp();
        if (lane == 0) tc5::mbar_arrive(bar(C::B_SE));    // the score slot may take the next tile
        const int col0 = t * 128;
        const bool need_mask = (p.causal && col0 + 127 > q0) || (col0 + 128 > p.seqlen);
        // 32-column chunks in which any row of this warp sees a key
        const int nch = need_mask ? min(4, (wlim - col0) / 32 + 1) : 4;
        const int rel = lim - col0;    // last visible column of this row
        float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};    // 4 / NA partial maxima for each accumulator
        if (need_mask) {
#pragma unroll
          for (int c = 0; c < 4; ++c)
            if (c < nch) {
#pragma unroll
              for (int i = 0; i < 32; ++i) {
                float& x = mx4[NA == 1 ? i & 3 : (c >> 1) * 2 + (i & 1)];
                if (c * 32 + i <= rel) x = fmaxf(x, __uint_as_float(r[c][i]));
              }
            }
        } else {
#pragma unroll
          for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int i = 0; i < 32; i += 2) {
              float& x = mx4[NA == 1 ? (i >> 1) & 3 : (c >> 1) * 2 + ((i >> 1) & 1)];
              x = max3(x, __uint_as_float(r[c][i]), __uint_as_float(r[c][i + 1]));
            }
        }
        const float lag = NA == 1 && t >= item.first + kExactTiles * item.step ? kRescaleStep : 0.0f;
        float corr[NA];
        bool rescale[NA];
        uint64_t nm2[NA];
#pragma unroll
        for (int a = 0; a < NA; ++a) {
          const float raw = NA == 1 ? fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) : fmaxf(mx4[2 * a], mx4[2 * a + 1]);
          const float mx = raw == -INFINITY ? -INFINITY : raw * sl;    // no visible key: whatever the sign of the scale
          const bool grow_m = mx > m[a] + lag || (m[a] == -INFINITY && mx > -INFINITY);
          corr[a] = 1.0f;
          rescale[a] = __any_sync(0xffffffffu, grow_m);
          if (grow_m) {
            corr[a] = (m[a] == -INFINITY) ? 0.0f : ex2(m[a] - mx);
            l[a] *= corr[a];
            m[a] = mx;
          }
          const float m_use = (m[a] == -INFINITY) ? 0.0f : m[a];
          nm2[a] = f2_pack(-m_use, -m_use);
        }
        // p = exp2(s * sl - m), two columns per multiply-add and per sum; masked columns are cleared afterwards
        uint64_t sum2[2] = {f2_pack(0.0f, 0.0f), f2_pack(0.0f, 0.0f)};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          if (c < nch) {
#pragma unroll
            for (int i = 0; i < 32; i += 2) {
              const float2 x = f2_unpack(f2_fma(f2_pack(__uint_as_float(r[c][i]), __uint_as_float(r[c][i + 1])), sl2, nm2[c * NA / 4]));
              r[c][i] = __float_as_uint(ex2(x.x));
              r[c][i + 1] = __float_as_uint(ex2(x.y));
            }
            if (need_mask) {
#pragma unroll
              for (int i = 0; i < 32; ++i)
                if (c * 32 + i > rel) r[c][i] = 0u;
            }
          } else {
#pragma unroll
            for (int i = 0; i < 32; ++i) r[c][i] = 0u;
          }
          // sums and packed probabilities of this chunk: columns 2j, 2j + 1 -> word 16 c + j
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            const float e0 = __uint_as_float(r[c][i]), e1 = __uint_as_float(r[c][i + 1]);
            uint64_t& x = sum2[NA == 1 ? (i >> 1) & 1 : c >> 1];
            x = f2_add(x, f2_pack(e0, e1));
            r[c >> 1][(c & 1) * 16 + (i >> 1)] = pack_bf16(e0, e1);
          }
        }
        const float2 sa = f2_unpack(sum2[0]), sb = f2_unpack(sum2[1]);
        if (NA == 1) {
          l[0] += (sa.x + sa.y) + (sb.x + sb.y);
        } else {
          l[0] += sa.x + sa.y;
          l[NA - 1] += sb.x + sb.y;
        }
        // P V of this group's previous tile is complete: P may be overwritten, O may be rescaled
        if (n > 0 && !wait_warp(bar(C::B_OF + wg), (n - 1) & 1u)) { ok = false; break; }
        tc5::fence_after_sync();
        tc5::tmem_st32(tp, r[0]);
        tc5::tmem_st32(tp + 32u, r[1]);
        if (t > item.first) {
#pragma unroll
          for (int a = 0; a < NA; ++a) {
            if (rescale[a]) {
              const uint64_t c2 = f2_pack(corr[a], corr[a]);
              uint32_t x[D / 32][32];    // all columns at once: one round trip to tensor memory
#pragma unroll
              for (int c = 0; c < D / 32; ++c) tc5::tmem_ld32(to + (uint32_t)(a * D + c * 32), x[c]);
              tc5::tmem_ld_wait();
#pragma unroll
              for (int c = 0; c < D / 32; ++c) {
#pragma unroll
                for (int i = 0; i < 32; i += 2) {
                  const float2 v = f2_unpack(f2_mul(f2_pack(__uint_as_float(x[c][i]), __uint_as_float(x[c][i + 1])), c2));
                  x[c][i] = __float_as_uint(v.x);
                  x[c][i + 1] = __float_as_uint(v.y);
                }
                tc5::tmem_st32(to + (uint32_t)(a * D + c * 32), x[c]);
              }
            }
          }
        }
        tc5::tmem_st_wait();
        tc5::fence_before_sync();
        __syncwarp();
        if (lane == 0) tc5::mbar_arrive(bar(C::B_PF + wg));
      }
      if (!ok || (n > 0 && !wait_warp(bar(C::B_OF + wg), (n - 1) & 1u))) { ok = false; break; }
      tc5::fence_after_sync();
      const int64_t lse_row = (int64_t)bh * p.seqlen + grow;
      __nv_bfloat16* dst = p.o + (int64_t)b * p.o_sb + (int64_t)(q0 + qd * 32) * p.o_ss + (int64_t)h * p.o_sh;    // the warp's first row
      const int rows = p.seqlen - q0 - qd * 32;    // of which exist
      // the row's maximum and sum over its accumulators, and the factor of each
      float mr = m[0], lr = l[0], f[NA];
      f[0] = 1.0f;
      if (NA == 2) {
        mr = fmaxf(m[0], m[NA - 1]);
        f[0] = (m[0] == -INFINITY) ? 0.0f : ex2(m[0] - mr);
        f[NA - 1] = (m[NA - 1] == -INFINITY) ? 0.0f : ex2(m[NA - 1] - mr);
        lr = l[0] * f[0] + l[NA - 1] * f[NA - 1];
      }
      if (!item.shared) {
        const float inv = lr > 0.0f ? 1.0f / lr : 0.0f;
#pragma unroll
        for (int c = 0; c < D; c += 64) {
          float v[64];
#pragma unroll
          for (int a = 0; a < NA; ++a) {
            uint32_t x[2][32];
            tc5::tmem_ld32(to + (uint32_t)(a * D + c), x[0]);
            tc5::tmem_ld32(to + (uint32_t)(a * D + c) + 32u, x[1]);
            tc5::tmem_ld_wait();
            const float fa = f[a] * inv;
#pragma unroll
            for (int i = 0; i < 64; ++i) v[i] = a ? fmaf(__uint_as_float(x[i >> 5][i & 31]), fa, v[i]) : __uint_as_float(x[i >> 5][i & 31]) * fa;
          }
          st_rows64(dst + c, p.o_ss, rows, v);
        }
        tc5::fence_before_sync();    // the next item's first P is handed over after these reads
        if (grow < p.seqlen) p.lse[lse_row] = lr > 0.0f ? mr * kLn2 + logf(lr) : -INFINITY;
      } else {
        // the last item of the CTA: maxima, sums and factors change hands through the P columns, which nothing uses any more
        uint32_t x[16] = {__float_as_uint(mr), __float_as_uint(lr), __float_as_uint(f[0]), __float_as_uint(f[NA - 1])}, y[16];
        tc5::tmem_st16(tp, x);
        tc5::tmem_st_wait();
        tc5::fence_before_sync();
        __syncwarp();
        if (lane == 0) tc5::mbar_arrive(bar(C::B_X));
        if (!wait_warp(bar(C::B_X), 0u)) { ok = false; break; }
        tc5::fence_after_sync();
        tc5::tmem_ld16(tlane + TM_P + (uint32_t)(wg ^ 1) * 64u, y);
        tc5::tmem_ld_wait();
        const float om = __uint_as_float(y[0]), ol = __uint_as_float(y[1]);
        const float m0 = wg ? om : mr, m1 = wg ? mr : om, l0 = wg ? ol : lr, l1 = wg ? lr : ol;
        const float mm = fmaxf(m0, m1);
        const float f0 = (m0 == -INFINITY) ? 0.0f : ex2(m0 - mm);
        const float f1 = (m1 == -INFINITY) ? 0.0f : ex2(m1 - mm);
        const float lt = l0 * f0 + l1 * f1;
        const float inv = lt > 0.0f ? 1.0f / lt : 0.0f;
        // each group stores every other 32 columns; an item of one tile has left the second stream's accumulators unwritten
#pragma unroll
        for (int c = 0; c < D; c += 64) {
          const uint32_t col = (uint32_t)(c + wg * 32);
          float v[32];
#pragma unroll
          for (int a = 0; a < NA; ++a) {
            const float own = f[a], others = __uint_as_float(y[a ? 3 : 2]);
            const float g0 = f0 * inv * (wg ? others : own), g1 = f1 * inv * (wg ? own : others);
            uint32_t a0[32], a1[32];
            tc5::tmem_ld32(tlane + TM_O + (uint32_t)(a * D) + col, a0);
            tc5::tmem_ld32(tlane + TM_O + 128u + (uint32_t)(a * D) + col, a1);
            tc5::tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) {
              const float o0 = __uint_as_float(a0[i]) * g0;
              v[i] = fmaf(n_t > 1 ? __uint_as_float(a1[i]) : 0.0f, g1, a ? v[i] + o0 : o0);
            }
          }
          if (row < p.seqlen - q0) st_row32(dst + (int64_t)lane * p.o_ss + col, v);
        }
        if (wg == 0 && grow < p.seqlen) p.lse[lse_row] = lt > 0.0f ? mm * kLn2 + logf(lt) : -INFINITY;
      }
    }
  }

  // ---------------------------------------------------------------------- tear-down
  __syncwarp();
  if (*abort_flag) __nanosleep(200000);    // let copies / MMAs in flight finish before smem and TMEM go away
  tc5::fence_before_sync();
  __syncthreads();
  tc5::fence_after_sync();
  if (warp == 1) tc5::tmem_dealloc(tmem_base, TM_COLS);
}

// ===================================================================================== delta = rowsum(dO * O)
struct DeltaParams {
  const __nv_bfloat16* o;
  const __nv_bfloat16* d_o;
  float* delta;
  int64_t o_sb, o_ss, o_sh, do_sb, do_ss, do_sh;
  int batch, heads, seqlen;
};

// Bound by memory: one pass over O and dO.  D / 8 lanes read one row with 16-byte loads and rows are taken in the order of
// their addresses ([batch, seq, head]), two per lane group, so that a warp keeps 2 KB of loads in flight.  A warp per row
// in [batch, head, seq] order, 8 bytes a lane, took 50 us for 4 x 2048 x 32 heads of 128 (134 MB); this takes 35 us.
template <int D>
__global__ void __launch_bounds__(256) attn_delta_tc_kernel(const DeltaParams p) {
  constexpr int L = D / 8;             // lanes of a row
  constexpr int ROWS = 256 / L;        // rows of a CTA and step
  const int sub = threadIdx.x % L;
  const int64_t total = (int64_t)p.batch * p.heads * p.seqlen;
  const int64_t r0 = (int64_t)blockIdx.x * (2 * ROWS) + threadIdx.x / L;
  Bytes16 a[2], g[2];
  int64_t out[2];
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const int64_t r = r0 + k * ROWS;
    a[k] = g[k] = Bytes16{};
    out[k] = -1;
    if (r < total) {
      const int h = (int)(r % p.heads);
      const int64_t bs = r / p.heads;
      const int s = (int)(bs % p.seqlen), b = (int)(bs / p.seqlen);
      a[k] = *reinterpret_cast<const Bytes16*>(p.o + (int64_t)b * p.o_sb + (int64_t)s * p.o_ss + (int64_t)h * p.o_sh + sub * 8);
      g[k] = *reinterpret_cast<const Bytes16*>(p.d_o + (int64_t)b * p.do_sb + (int64_t)s * p.do_ss + (int64_t)h * p.do_sh + sub * 8);
      out[k] = ((int64_t)b * p.heads + h) * p.seqlen + s;
    }
  }
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const __nv_bfloat162* a2 = reinterpret_cast<const __nv_bfloat162*>(&a[k]);
    const __nv_bfloat162* g2 = reinterpret_cast<const __nv_bfloat162*>(&g[k]);
    float acc = 0.0f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 x = __bfloat1622float2(a2[i]);
      const float2 y = __bfloat1622float2(g2[i]);
      acc = fmaf(x.x, y.x, fmaf(x.y, y.y, acc));
    }
#pragma unroll
    for (int o = L / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (sub == 0 && out[k] >= 0) p.delta[out[k]] = acc;
  }
}

// ============================================================================================ dK / dV
namespace dkv {
constexpr uint32_t PANEL_KV = 128 * 128;    // [128 key rows][64 bf16]
constexpr uint32_t TILE_KV = 2 * PANEL_KV;
constexpr uint32_t PANEL_Q = 64 * 128;      // [64 query rows][64 bf16]
constexpr uint32_t TILE_Q = 2 * PANEL_Q;    // 16 KB
constexpr uint32_t TILE_P = 128 * 128;      // [128 key rows][64 queries] bf16
constexpr int NSQ = 3;    // ring of Q/dO stages: a stage is read by the first and by the last MMA of its tile
constexpr uint32_t OFF_K = 0, OFF_V = TILE_KV, OFF_Q = 2 * TILE_KV, OFF_DO = OFF_Q + NSQ * TILE_Q, OFF_PT = OFF_DO + NSQ * TILE_Q,
                   OFF_DST = OFF_PT + 2 * TILE_P, OFF_LSE = OFF_DST + 2 * TILE_P, OFF_BAR = OFF_LSE + NSQ * 2 * 64 * 4;
enum { B_KV = 0, B_QF = 1, B_QE = B_QF + NSQ, B_SF = B_QE + NSQ, B_SE = B_SF + 2, B_PF = B_SE + 2, B_PE = B_PF + 2, B_ACC = B_PE + 2,
       NBAR = B_ACC + 1 };
constexpr int SMEM = OFF_BAR + NBAR * 8 + 16 + 1024;
constexpr uint32_t TM_ST = 0, TM_DPT = 128, TM_DV = 256, TM_DK = 384, TM_COLS = 512;
}    // namespace dkv

__global__ void __launch_bounds__(kTcThreads, 1)
attn_bwd_dkdv_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                        const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_do, const TcParams p) {
  using namespace dkv;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = tc5::smem_u32(smem_raw);
  const uint32_t base = (raw_addr + 1023u) & ~1023u;
  uint8_t* smem = smem_raw + (base - raw_addr);
  const uint32_t bars = base + OFF_BAR;
  auto bar = [&](int i) { return bars + 8u * (uint32_t)i; };
  float* s_lse = reinterpret_cast<float*>(smem + OFF_LSE);    // [NSQ][64] log2-scaled lse, then [NSQ][64] delta
  float* s_delta = s_lse + NSQ * 64;
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(smem + OFF_BAR + NBAR * 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);
  // Wait used by full warps that go on to warp-collective TMEM accesses: the outcome is made uniform.
  auto wait_warp = [&](uint32_t br, uint32_t ph) {
    return __all_sync(0xffffffffu, tc5::mbar_wait(br, ph, abort_flag, p.status, kStatusBit)) != 0;
  };

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int kt = blockIdx.x;    // key tile 0 has the most query tiles under a causal mask and starts first
  const int bh = blockIdx.y;
  const int b = bh / p.heads;
  const int h = bh - b * p.heads;
  const int k0 = kt * 128;
  const int nq_all = (p.seqlen + 63) / 64;
  const int t_first = p.causal ? 2 * kt : 0;
  const int n_q = nq_all - t_first;    // >= 1 because k0 < seqlen

  if (threadIdx.x == 0) {
    tc5::mbar_init(bar(B_KV), 1);
    for (int s = 0; s < NSQ; ++s) {
      tc5::mbar_init(bar(B_QF + s), 2);    // TMA bytes + the lse/delta rows written by warp 0
      tc5::mbar_init(bar(B_QE + s), 5);    // last MMA that reads the stage + four softmax warps
    }
    for (int s = 0; s < 2; ++s) {
      tc5::mbar_init(bar(B_SF + s), 1);
      tc5::mbar_init(bar(B_SE + s), 4);
      tc5::mbar_init(bar(B_PF + s), 4);
      tc5::mbar_init(bar(B_PE + s), 1);
    }
    tc5::mbar_init(bar(B_ACC), 1);
    *abort_flag = 0;
    tc5::mbar_fence_init();
    tc5::tma_prefetch_desc(&map_q);
    tc5::tma_prefetch_desc(&map_k);
    tc5::tma_prefetch_desc(&map_v);
    tc5::tma_prefetch_desc(&map_do);
  }
  if (warp == 1) {
    tc5::tmem_alloc(tc5::smem_u32(tmem_holder), TM_COLS);
    tc5::tmem_relinquish();
  }
  tc5::fence_before_sync();
  __syncthreads();
  tc5::fence_after_sync();
  const uint32_t tmem_base = *tmem_holder;

  if (warp == 0) {
    // ------------------------------------------------------------------ producer (whole warp: lane 0 issues TMA)
    if (lane == 0) {
      tc5::mbar_arrive_expect_tx(bar(B_KV), 2 * TILE_KV);
      tc5::tma_load_4d(base + OFF_K, &map_k, 0, h, k0, b, bar(B_KV));
      tc5::tma_load_4d(base + OFF_K + PANEL_KV, &map_k, 64, h, k0, b, bar(B_KV));
      tc5::tma_load_4d(base + OFF_V, &map_v, 0, h, k0, b, bar(B_KV));
      tc5::tma_load_4d(base + OFF_V + PANEL_KV, &map_v, 64, h, k0, b, bar(B_KV));
    }
    const float* glse = p.lse + (int64_t)bh * p.seqlen;
    const float* gdelta = p.delta + (int64_t)bh * p.seqlen;
    for (int t = 0; t < n_q; ++t) {
      const int s = t % NSQ;
      const uint32_t ph = (uint32_t)(t / NSQ) & 1u;
      const int qrow0 = (t_first + t) * 64;
      TC_WAIT(bar(B_QE + s), ph ^ 1u);
      if (lane == 0) {
        tc5::mbar_arrive_expect_tx(bar(B_QF + s), 2 * TILE_Q);
        tc5::tma_load_4d(base + OFF_Q + s * TILE_Q, &map_q, 0, h, qrow0, b, bar(B_QF + s));
        tc5::tma_load_4d(base + OFF_Q + s * TILE_Q + PANEL_Q, &map_q, 64, h, qrow0, b, bar(B_QF + s));
        tc5::tma_load_4d(base + OFF_DO + s * TILE_Q, &map_do, 0, h, qrow0, b, bar(B_QF + s));
        tc5::tma_load_4d(base + OFF_DO + s * TILE_Q + PANEL_Q, &map_do, 64, h, qrow0, b, bar(B_QF + s));
      }
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int r = lane + 32 * i;
        const bool in = qrow0 + r < p.seqlen;
        s_lse[s * 64 + r] = in ? glse[qrow0 + r] * kLog2e : INFINITY;    // +inf makes the probability exactly zero
        s_delta[s * 64 + r] = in ? gdelta[qrow0 + r] : 0.0f;
      }
      __syncwarp();
      if (lane == 0) tc5::mbar_arrive(bar(B_QF + s));
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (lane == 0) {
      const uint32_t idesc_s = tc5::idesc_bf16(128, 64, 0, 0);
      const uint32_t idesc_acc = tc5::idesc_bf16(128, 128, 0, 1);
      // S^T = K Q_t^T and dP^T = V dO_t^T into buffer t&1
      auto issue_s = [&](int t) -> bool {
        const int s = t & 1;
        const uint32_t ph = (uint32_t)(t >> 1) & 1u;
        const int st = t % NSQ;
        if (!tc5::mbar_wait(bar(B_SE + s), ph ^ 1u, abort_flag, p.status, kStatusBit)) return false;
        if (!tc5::mbar_wait(bar(B_QF + st), (uint32_t)(t / NSQ) & 1u, abort_flag, p.status, kStatusBit)) return false;
        tc5::fence_after_sync();
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
          const uint32_t offa = (uint32_t)(kk >> 2) * PANEL_KV + (uint32_t)(kk & 3) * 32u;
          const uint32_t offb = (uint32_t)(kk >> 2) * PANEL_Q + (uint32_t)(kk & 3) * 32u;
          tc5::mma_f16(tmem_base + TM_ST + (uint32_t)s * 64u, tc5::smem_desc_k_sw128(base + OFF_K + offa),
                       tc5::smem_desc_k_sw128(base + OFF_Q + st * TILE_Q + offb), idesc_s, kk ? 1u : 0u);
        }
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
          const uint32_t offa = (uint32_t)(kk >> 2) * PANEL_KV + (uint32_t)(kk & 3) * 32u;
          const uint32_t offb = (uint32_t)(kk >> 2) * PANEL_Q + (uint32_t)(kk & 3) * 32u;
          tc5::mma_f16(tmem_base + TM_DPT + (uint32_t)s * 64u, tc5::smem_desc_k_sw128(base + OFF_V + offa),
                       tc5::smem_desc_k_sw128(base + OFF_DO + st * TILE_Q + offb), idesc_s, kk ? 1u : 0u);
        }
        tc5::mma_commit(bar(B_SF + s));
        return true;
      };
      do {
        TC_WAIT(bar(B_KV), 0u);
        if (!issue_s(0)) break;
        if (n_q > 1 && !issue_s(1)) break;
        bool ok = true;
        for (int t = 0; t < n_q; ++t) {
          // the scores two tiles ahead go first: their buffer was released as soon as tile t had been read
          if (t + 2 < n_q && !issue_s(t + 2)) { ok = false; break; }
          const int s = t & 1;
          const int st = t % NSQ;
          const uint32_t ph = (uint32_t)(t >> 1) & 1u;
          if (!tc5::mbar_wait(bar(B_PF + s), ph, abort_flag, p.status, kStatusBit)) { ok = false; break; }
          tc5::fence_after_sync();
          // dV += P^T dO_t ; dK += dS^T Q_t : A from the softmax threads (K-major), B = the TMA tile read MN-major
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) {
            tc5::mma_f16(tmem_base + TM_DV, tc5::smem_desc_k_sw128(base + OFF_PT + s * TILE_P + (uint32_t)kk * 32u),
                         tc5::smem_desc_mn_sw128(base + OFF_DO + st * TILE_Q + (uint32_t)kk * 2048u, PANEL_Q), idesc_acc,
                         (t | kk) ? 1u : 0u);
          }
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) {
            tc5::mma_f16(tmem_base + TM_DK, tc5::smem_desc_k_sw128(base + OFF_DST + s * TILE_P + (uint32_t)kk * 32u),
                         tc5::smem_desc_mn_sw128(base + OFF_Q + st * TILE_Q + (uint32_t)kk * 2048u, PANEL_Q), idesc_acc,
                         (t | kk) ? 1u : 0u);
          }
          tc5::mma_commit(bar(B_PE + s));
          tc5::mma_commit(bar(B_QE + st));
        }
        if (ok) tc5::mma_commit(bar(B_ACC));
      } while (false);
    }
  } else {
    // ------------------------------------------------------------------ one thread per key row
    const int qd = warp & 3;
    const int wg = (warp - 2) >> 2;    // group 0 takes the even query tiles (buffer 0), group 1 the odd ones
    const int row = qd * 32 + lane;
    const int grow = k0 + row;
    const uint32_t tlane = tmem_base + ((uint32_t)(qd * 32) << 16);
    const float sl = p.scale * kLog2e;
    bool ok = true;
    for (int t = wg; t < n_q; t += 2) {
      const int s = t & 1;
      const int st = t % NSQ;
      const uint32_t ph = (uint32_t)(t >> 1) & 1u;
      const int qrow0 = (t_first + t) * 64;
      if (!wait_warp(bar(B_QF + st), (uint32_t)(t / NSQ) & 1u)) { ok = false; break; }
      if (!wait_warp(bar(B_SF + s), ph)) { ok = false; break; }
      tc5::fence_after_sync();
      const bool need_mask = p.causal && (qrow0 < k0 + 128);
      const float4* lse2 = reinterpret_cast<const float4*>(s_lse + st * 64);
      const float4* dlt = reinterpret_cast<const float4*>(s_delta + st * 64);
      uint32_t rs[2][32], rd[2][32];
      tc5::tmem_ld32(tlane + TM_ST + (uint32_t)s * 64u, rs[0]);
      tc5::tmem_ld32(tlane + TM_ST + (uint32_t)s * 64u + 32u, rs[1]);
      tc5::tmem_ld32(tlane + TM_DPT + (uint32_t)s * 64u, rd[0]);
      tc5::tmem_ld32(tlane + TM_DPT + (uint32_t)s * 64u + 32u, rd[1]);
      tc5::tmem_ld_wait();
      tc5::fence_before_sync();
      __syncwarp();
      if (lane == 0) tc5::mbar_arrive(bar(B_SE + s));    // the buffer may take tile t + 2
      if (!wait_warp(bar(B_PE + s), ph ^ 1u)) { ok = false; break; }
      const uint32_t prow = base + OFF_PT + s * TILE_P + (uint32_t)row * 128u;
      const uint32_t drow = base + OFF_DST + s * TILE_P + (uint32_t)row * 128u;
      const uint32_t swz = (uint32_t)(row & 7);
#pragma unroll
      for (int g = 0; g < 8; ++g) {    // 16-byte chunk g = queries 8g .. 8g+7 of the tile
        float e[8], ds[8];
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
          const float4 l4 = lse2[g * 2 + hh];
          const float4 d4 = dlt[g * 2 + hh];
          const float la[4] = {l4.x, l4.y, l4.z, l4.w};
          const float da[4] = {d4.x, d4.y, d4.z, d4.w};
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int i = hh * 4 + u;
            const int ql = g * 8 + i;
            float ev = ex2(fmaf(__uint_as_float(rs[ql >> 5][ql & 31]), sl, -la[u]));
            if (need_mask && qrow0 + ql < grow) ev = 0.0f;
            e[i] = ev;
            ds[i] = ev * (__uint_as_float(rd[ql >> 5][ql & 31]) - da[u]);
          }
        }
        const uint32_t off = (((uint32_t)g) ^ swz) << 4;
        st_shared_v4(prow + off, pack_bf16(e[0], e[1]), pack_bf16(e[2], e[3]), pack_bf16(e[4], e[5]), pack_bf16(e[6], e[7]));
        st_shared_v4(drow + off, pack_bf16(ds[0], ds[1]), pack_bf16(ds[2], ds[3]), pack_bf16(ds[4], ds[5]), pack_bf16(ds[6], ds[7]));
      }
      tc5::fence_before_sync();
      fence_async_smem();
      __syncwarp();
      if (lane == 0) {
        tc5::mbar_arrive(bar(B_PF + s));
        tc5::mbar_arrive(bar(B_QE + st));
      }
    }
    if (ok && wait_warp(bar(B_ACC), 0u)) {
      tc5::fence_after_sync();
      __nv_bfloat16* dv = p.dv + (int64_t)b * p.dv_sb + (int64_t)grow * p.dv_ss + (int64_t)h * p.dv_sh;
      __nv_bfloat16* dk = p.dk + (int64_t)b * p.dk_sb + (int64_t)grow * p.dk_ss + (int64_t)h * p.dk_sh;
      // group 0 stores dV, group 1 stores dK
      __nv_bfloat16* dst = wg == 0 ? dv : dk;
      const float f = wg == 0 ? 1.0f : p.scale;
      const uint32_t tsrc = tlane + (wg == 0 ? TM_DV : TM_DK);
#pragma unroll
      for (int c = 0; c < 4; c += 2) {
        uint32_t r0[32], r1[32];
        float v[32];
        tc5::tmem_ld32(tsrc + (uint32_t)c * 32u, r0);
        tc5::tmem_ld32(tsrc + (uint32_t)c * 32u + 32u, r1);
        tc5::tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r0[i]) * f;
        if (grow < p.seqlen) st_row32(dst + c * 32, v);
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r1[i]) * f;
        if (grow < p.seqlen) st_row32(dst + c * 32 + 32, v);
      }
    }
  }

  __syncwarp();
  if (*abort_flag) __nanosleep(200000);
  tc5::fence_before_sync();
  __syncthreads();
  tc5::fence_after_sync();
  if (warp == 1) tc5::tmem_dealloc(tmem_base, TM_COLS);
}

// ================================================================================================= dQ
namespace dqk {
constexpr uint32_t PANEL_Q = 128 * 128;     // [128 query rows][64 bf16]
constexpr uint32_t TILE_Q = 2 * PANEL_Q;
constexpr uint32_t PANEL_KV = 64 * 128;     // [64 key rows][64 bf16]
constexpr uint32_t TILE_KV = 2 * PANEL_KV;
constexpr uint32_t TILE_DS = 128 * 128;     // [128 query rows][64 keys] bf16
constexpr int NSK = 4;    // ring of K/V stages: a stage is read by the first and by the last MMA of its tile
constexpr uint32_t OFF_Q = 0, OFF_DO = TILE_Q, OFF_K = 2 * TILE_Q, OFF_V = OFF_K + NSK * TILE_KV, OFF_DS = OFF_V + NSK * TILE_KV,
                   OFF_BAR = OFF_DS + 2 * TILE_DS;
enum { B_Q = 0, B_KF = 1, B_KE = B_KF + NSK, B_SF = B_KE + NSK, B_SE = B_SF + 2, B_PF = B_SE + 2, B_PE = B_PF + 2, B_ACC = B_PE + 2,
       NBAR = B_ACC + 1 };
constexpr int SMEM = OFF_BAR + NBAR * 8 + 16 + 1024;
constexpr uint32_t TM_S = 0, TM_DP = 128, TM_DQ = 256, TM_COLS = 512;
}    // namespace dqk

__global__ void __launch_bounds__(kTcThreads, 1)
attn_bwd_dq_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                      const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_do, const TcParams p) {
  using namespace dqk;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = tc5::smem_u32(smem_raw);
  const uint32_t base = (raw_addr + 1023u) & ~1023u;
  uint8_t* smem = smem_raw + (base - raw_addr);
  const uint32_t bars = base + OFF_BAR;
  auto bar = [&](int i) { return bars + 8u * (uint32_t)i; };
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(smem + OFF_BAR + NBAR * 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);
  // Wait used by full warps that go on to warp-collective TMEM accesses: the outcome is made uniform.
  auto wait_warp = [&](uint32_t br, uint32_t ph) {
    return __all_sync(0xffffffffu, tc5::mbar_wait(br, ph, abort_flag, p.status, kStatusBit)) != 0;
  };

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int qt = (int)gridDim.x - 1 - (int)blockIdx.x;
  const int bh = blockIdx.y;
  const int b = bh / p.heads;
  const int h = bh - b * p.heads;
  const int q0 = qt * 128;
  const int nk_all = (p.seqlen + 63) / 64;
  const int n_kv = p.causal ? min(2 * qt + 2, nk_all) : nk_all;

  if (threadIdx.x == 0) {
    tc5::mbar_init(bar(B_Q), 1);
    for (int s = 0; s < NSK; ++s) {
      tc5::mbar_init(bar(B_KF + s), 1);
      tc5::mbar_init(bar(B_KE + s), 1);
    }
    for (int s = 0; s < 2; ++s) {
      tc5::mbar_init(bar(B_SF + s), 1);
      tc5::mbar_init(bar(B_SE + s), 4);
      tc5::mbar_init(bar(B_PF + s), 4);
      tc5::mbar_init(bar(B_PE + s), 1);
    }
    tc5::mbar_init(bar(B_ACC), 1);
    *abort_flag = 0;
    tc5::mbar_fence_init();
    tc5::tma_prefetch_desc(&map_q);
    tc5::tma_prefetch_desc(&map_k);
    tc5::tma_prefetch_desc(&map_v);
    tc5::tma_prefetch_desc(&map_do);
  }
  if (warp == 1) {
    tc5::tmem_alloc(tc5::smem_u32(tmem_holder), TM_COLS);
    tc5::tmem_relinquish();
  }
  tc5::fence_before_sync();
  __syncthreads();
  tc5::fence_after_sync();
  const uint32_t tmem_base = *tmem_holder;

  if (warp == 0) {
    if (lane == 0) {
      tc5::mbar_arrive_expect_tx(bar(B_Q), 2 * TILE_Q);
      tc5::tma_load_4d(base + OFF_Q, &map_q, 0, h, q0, b, bar(B_Q));
      tc5::tma_load_4d(base + OFF_Q + PANEL_Q, &map_q, 64, h, q0, b, bar(B_Q));
      tc5::tma_load_4d(base + OFF_DO, &map_do, 0, h, q0, b, bar(B_Q));
      tc5::tma_load_4d(base + OFF_DO + PANEL_Q, &map_do, 64, h, q0, b, bar(B_Q));
      for (int j = 0; j < n_kv; ++j) {
        const int s = j % NSK;
        const uint32_t ph = (uint32_t)(j / NSK) & 1u;
        TC_WAIT(bar(B_KE + s), ph ^ 1u);
        tc5::mbar_arrive_expect_tx(bar(B_KF + s), 2 * TILE_KV);
        tc5::tma_load_4d(base + OFF_K + s * TILE_KV, &map_k, 0, h, j * 64, b, bar(B_KF + s));
        tc5::tma_load_4d(base + OFF_K + s * TILE_KV + PANEL_KV, &map_k, 64, h, j * 64, b, bar(B_KF + s));
        tc5::tma_load_4d(base + OFF_V + s * TILE_KV, &map_v, 0, h, j * 64, b, bar(B_KF + s));
        tc5::tma_load_4d(base + OFF_V + s * TILE_KV + PANEL_KV, &map_v, 64, h, j * 64, b, bar(B_KF + s));
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      const uint32_t idesc_s = tc5::idesc_bf16(128, 64, 0, 0);
      const uint32_t idesc_acc = tc5::idesc_bf16(128, 128, 0, 1);
      auto issue_s = [&](int j) -> bool {
        const int s = j & 1;
        const int st = j % NSK;
        const uint32_t ph = (uint32_t)(j >> 1) & 1u;
        if (!tc5::mbar_wait(bar(B_SE + s), ph ^ 1u, abort_flag, p.status, kStatusBit)) return false;
        if (!tc5::mbar_wait(bar(B_KF + st), (uint32_t)(j / NSK) & 1u, abort_flag, p.status, kStatusBit)) return false;
        tc5::fence_after_sync();
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
          const uint32_t offa = (uint32_t)(kk >> 2) * PANEL_Q + (uint32_t)(kk & 3) * 32u;
          const uint32_t offb = (uint32_t)(kk >> 2) * PANEL_KV + (uint32_t)(kk & 3) * 32u;
          tc5::mma_f16(tmem_base + TM_S + (uint32_t)s * 64u, tc5::smem_desc_k_sw128(base + OFF_Q + offa),
                       tc5::smem_desc_k_sw128(base + OFF_K + st * TILE_KV + offb), idesc_s, kk ? 1u : 0u);
        }
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
          const uint32_t offa = (uint32_t)(kk >> 2) * PANEL_Q + (uint32_t)(kk & 3) * 32u;
          const uint32_t offb = (uint32_t)(kk >> 2) * PANEL_KV + (uint32_t)(kk & 3) * 32u;
          tc5::mma_f16(tmem_base + TM_DP + (uint32_t)s * 64u, tc5::smem_desc_k_sw128(base + OFF_DO + offa),
                       tc5::smem_desc_k_sw128(base + OFF_V + st * TILE_KV + offb), idesc_s, kk ? 1u : 0u);
        }
        tc5::mma_commit(bar(B_SF + s));
        return true;
      };
      do {
        TC_WAIT(bar(B_Q), 0u);
        if (!issue_s(0)) break;
        if (n_kv > 1 && !issue_s(1)) break;
        bool ok = true;
        for (int j = 0; j < n_kv; ++j) {
          // the scores two tiles ahead go first: their buffer was released as soon as tile j had been read
          if (j + 2 < n_kv && !issue_s(j + 2)) { ok = false; break; }
          const int s = j & 1;
          const int st = j % NSK;
          const uint32_t ph = (uint32_t)(j >> 1) & 1u;
          if (!tc5::mbar_wait(bar(B_PF + s), ph, abort_flag, p.status, kStatusBit)) { ok = false; break; }
          tc5::fence_after_sync();
          // dQ += dS K_j : B = the K tile with the key index as rows (MN-major)
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) {
            tc5::mma_f16(tmem_base + TM_DQ, tc5::smem_desc_k_sw128(base + OFF_DS + s * TILE_DS + (uint32_t)kk * 32u),
                         tc5::smem_desc_mn_sw128(base + OFF_K + st * TILE_KV + (uint32_t)kk * 2048u, PANEL_KV), idesc_acc,
                         (j | kk) ? 1u : 0u);
          }
          tc5::mma_commit(bar(B_PE + s));
          tc5::mma_commit(bar(B_KE + st));
        }
        if (ok) tc5::mma_commit(bar(B_ACC));
      } while (false);
    }
  } else {
    const int qd = warp & 3;
    const int wg = (warp - 2) >> 2;    // group 0 takes the even key tiles (buffer 0), group 1 the odd ones
    const int row = qd * 32 + lane;
    const int grow = q0 + row;
    const uint32_t tlane = tmem_base + ((uint32_t)(qd * 32) << 16);
    const float sl = p.scale * kLog2e;
    const bool in = grow < p.seqlen;
    const float lse2 = in ? p.lse[(int64_t)bh * p.seqlen + grow] * kLog2e : INFINITY;
    const float dlt = in ? p.delta[(int64_t)bh * p.seqlen + grow] : 0.0f;
    const int lim = p.causal ? min(grow, p.seqlen - 1) : p.seqlen - 1;
    bool ok = true;
    for (int j = wg; j < n_kv; j += 2) {
      const int s = j & 1;
      const uint32_t ph = (uint32_t)(j >> 1) & 1u;
      const int col0 = j * 64;
      if (!wait_warp(bar(B_SF + s), ph)) { ok = false; break; }
      tc5::fence_after_sync();
      const bool need_mask = (p.causal && col0 + 63 > q0) || (col0 + 64 > p.seqlen);
      uint32_t rs[2][32], rd[2][32];
      tc5::tmem_ld32(tlane + TM_S + (uint32_t)s * 64u, rs[0]);
      tc5::tmem_ld32(tlane + TM_S + (uint32_t)s * 64u + 32u, rs[1]);
      tc5::tmem_ld32(tlane + TM_DP + (uint32_t)s * 64u, rd[0]);
      tc5::tmem_ld32(tlane + TM_DP + (uint32_t)s * 64u + 32u, rd[1]);
      tc5::tmem_ld_wait();
      tc5::fence_before_sync();
      __syncwarp();
      if (lane == 0) tc5::mbar_arrive(bar(B_SE + s));    // the buffer may take tile j + 2
      if (!wait_warp(bar(B_PE + s), ph ^ 1u)) { ok = false; break; }
      const uint32_t drow = base + OFF_DS + s * TILE_DS + (uint32_t)row * 128u;
      const uint32_t swz = (uint32_t)(row & 7);
#pragma unroll
      for (int g = 0; g < 8; ++g) {    // 16-byte chunk g = keys 8g .. 8g+7 of the tile
        float ds[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int c = g * 8 + i;
          float e = ex2(fmaf(__uint_as_float(rs[c >> 5][c & 31]), sl, -lse2));
          if (need_mask && col0 + c > lim) e = 0.0f;
          ds[i] = e * (__uint_as_float(rd[c >> 5][c & 31]) - dlt);
        }
        st_shared_v4(drow + ((((uint32_t)g) ^ swz) << 4), pack_bf16(ds[0], ds[1]), pack_bf16(ds[2], ds[3]), pack_bf16(ds[4], ds[5]),
                     pack_bf16(ds[6], ds[7]));
      }
      tc5::fence_before_sync();
      fence_async_smem();
      __syncwarp();
      if (lane == 0) tc5::mbar_arrive(bar(B_PF + s));
    }
    if (ok && wait_warp(bar(B_ACC), 0u)) {
      tc5::fence_after_sync();
      __nv_bfloat16* dq = p.dq + (int64_t)b * p.dq_sb + (int64_t)grow * p.dq_ss + (int64_t)h * p.dq_sh;
      // each group stores one half of the row
      uint32_t r0[32], r1[32];
      float v[32];
      tc5::tmem_ld32(tlane + TM_DQ + (uint32_t)wg * 64u, r0);
      tc5::tmem_ld32(tlane + TM_DQ + (uint32_t)wg * 64u + 32u, r1);
      tc5::tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r0[i]) * p.scale;
      if (in) st_row32(dq + wg * 64, v);
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r1[i]) * p.scale;
      if (in) st_row32(dq + wg * 64 + 32, v);
    }
  }

  __syncwarp();
  if (*abort_flag) __nanosleep(200000);
  tc5::fence_before_sync();
  __syncthreads();
  tc5::fence_after_sync();
  if (warp == 1) tc5::tmem_dealloc(tmem_base, TM_COLS);
}

// ========================================================================= dK / dV, 128-query tiles, dS^T in tensor memory
namespace dkv2 {
constexpr uint32_t PANEL = 128 * 128;      // [128 rows][64 bf16]
constexpr uint32_t TILE = 2 * PANEL;       // 32 KB: 128 rows x 128 bf16
constexpr int NSQ = 2;                     // Q / dO stages (a stage is read by the first and by the last MMA of its tile)
constexpr uint32_t OFF_K = 0, OFF_V = TILE, OFF_Q = 2 * TILE, OFF_DO = OFF_Q + NSQ * TILE, OFF_PT = OFF_DO + NSQ * TILE,
                   OFF_LSE = OFF_PT + TILE, OFF_BAR = OFF_LSE + NSQ * 2 * 128 * 4;
enum { B_KV = 0, B_QF = 1, B_QE = B_QF + NSQ, B_SF = B_QE + NSQ, B_SE = B_SF + 1, B_DF = B_SE + 1, B_PF = B_DF + 1, B_PE = B_PF + 1,
       B_ACC = B_PE + 1, NBAR = B_ACC + 1 };
// seven 32 KB tiles leave 3 KB of the 227 KB: the dynamic array is declared 128-byte aligned, so rounding its start up to
// 1024 bytes costs at most 896
constexpr int SMEM = OFF_BAR + NBAR * 8 + 16 + 896;
static_assert(SMEM <= 227 * 1024, "dK/dV kernel: shared memory");
constexpr uint32_t TM_ST = 0, TM_DPT = 128, TM_DV = 256, TM_DK = 384, TM_COLS = 512;
}    // namespace dkv2

// dK and dV for 128 key rows; query tiles of 128, so that S^T = K Q^T and dP^T = V dO^T are N = 128 products (an M = 128
// bf16 MMA costs the same for N = 64).  Tensor memory holds exactly S^T, dP^T, dV and dK (4 x 128 columns).  The eight
// softmax warps split a tile by columns (group g: queries 64 g .. 64 g + 63).  S^T is read into registers and released
// at once, so the scores of the next tile are computed during the arithmetic of this one; P^T goes to shared memory (A
// operand of dV += P^T dO); dS^T is packed to bf16 and stored over the dP^T columns it came from (A operand of
// dK += dS^T Q, read from tensor memory).  dP^T of the next tile is issued after dK of this one (in-order tensor pipe).
__global__ void __launch_bounds__(kTcThreads, 1)
attn_bwd_dkdv_tm_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                        const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_do, const TcParams p) {
  using namespace dkv2;
  extern __shared__ __align__(128) uint8_t smem_raw128[];
  const uint32_t raw_addr = tc5::smem_u32(smem_raw128);
  const uint32_t base = (raw_addr + 1023u) & ~1023u;
  uint8_t* smem = smem_raw128 + (base - raw_addr);
  const uint32_t bars = base + OFF_BAR;
  auto bar = [&](int i) { return bars + 8u * (uint32_t)i; };
  float* s_lse = reinterpret_cast<float*>(smem + OFF_LSE);    // [NSQ][128] log2-scaled lse, then [NSQ][128] delta
  float* s_delta = s_lse + NSQ * 128;
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(smem + OFF_BAR + NBAR * 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);
  auto wait_warp = [&](uint32_t br, uint32_t ph) {
    return __all_sync(0xffffffffu, tc5::mbar_wait(br, ph, abort_flag, p.status, kStatusBit)) != 0;
  };

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int kt = blockIdx.x;    // key tile 0 has the most query tiles under a causal mask and starts first
  const int bh = blockIdx.y;
  const int b = bh / p.heads;
  const int h = bh - b * p.heads;
  const int k0 = kt * 128;
  const int nq_all = (p.seqlen + 127) / 128;
  const int t_first = p.causal ? kt : 0;
  const int n_q = nq_all - t_first;    // >= 1 because k0 < seqlen

  if (threadIdx.x == 0) {
    tc5::mbar_init(bar(B_KV), 1);
    for (int s = 0; s < NSQ; ++s) {
      tc5::mbar_init(bar(B_QF + s), 2);    // TMA bytes + the lse/delta rows written by warp 0
      tc5::mbar_init(bar(B_QE + s), 9);    // last MMA that reads the stage + eight softmax warps
    }
    tc5::mbar_init(bar(B_SF), 1);
    tc5::mbar_init(bar(B_SE), 8);
    tc5::mbar_init(bar(B_DF), 1);
    tc5::mbar_init(bar(B_PF), 8);
    tc5::mbar_init(bar(B_PE), 1);
    tc5::mbar_init(bar(B_ACC), 1);
    *abort_flag = 0;
    tc5::mbar_fence_init();
    tc5::tma_prefetch_desc(&map_q);
    tc5::tma_prefetch_desc(&map_k);
    tc5::tma_prefetch_desc(&map_v);
    tc5::tma_prefetch_desc(&map_do);
  }
  if (warp == 1) {
    tc5::tmem_alloc(tc5::smem_u32(tmem_holder), TM_COLS);
    tc5::tmem_relinquish();
  }
  tc5::fence_before_sync();
  __syncthreads();
  tc5::fence_after_sync();
  const uint32_t tmem_base = *tmem_holder;

  if (warp == 0) {
    // ------------------------------------------------------------------ producer (whole warp: lane 0 issues TMA)
    if (lane == 0) {
      tc5::mbar_arrive_expect_tx(bar(B_KV), 2 * TILE);
      tc5::tma_load_4d(base + OFF_K, &map_k, 0, h, k0, b, bar(B_KV));
      tc5::tma_load_4d(base + OFF_K + PANEL, &map_k, 64, h, k0, b, bar(B_KV));
      tc5::tma_load_4d(base + OFF_V, &map_v, 0, h, k0, b, bar(B_KV));
      tc5::tma_load_4d(base + OFF_V + PANEL, &map_v, 64, h, k0, b, bar(B_KV));
    }
    const float* glse = p.lse + (int64_t)bh * p.seqlen;
    const float* gdelta = p.delta + (int64_t)bh * p.seqlen;
    for (int t = 0; t < n_q; ++t) {
      const int s = t % NSQ;
      const uint32_t ph = (uint32_t)(t / NSQ) & 1u;
      const int qrow0 = (t_first + t) * 128;
      TC_WAIT(bar(B_QE + s), ph ^ 1u);
      if (lane == 0) {
        tc5::mbar_arrive_expect_tx(bar(B_QF + s), 2 * TILE);
        tc5::tma_load_4d(base + OFF_Q + s * TILE, &map_q, 0, h, qrow0, b, bar(B_QF + s));
        tc5::tma_load_4d(base + OFF_Q + s * TILE + PANEL, &map_q, 64, h, qrow0, b, bar(B_QF + s));
        tc5::tma_load_4d(base + OFF_DO + s * TILE, &map_do, 0, h, qrow0, b, bar(B_QF + s));
        tc5::tma_load_4d(base + OFF_DO + s * TILE + PANEL, &map_do, 64, h, qrow0, b, bar(B_QF + s));
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = lane + 32 * i;
        const bool in = qrow0 + r < p.seqlen;
        s_lse[s * 128 + r] = in ? glse[qrow0 + r] * kLog2e : INFINITY;    // +inf makes the probability exactly zero
        s_delta[s * 128 + r] = in ? gdelta[qrow0 + r] : 0.0f;
      }
      __syncwarp();
      if (lane == 0) tc5::mbar_arrive(bar(B_QF + s));
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (lane == 0) {
      const uint32_t idesc_s = tc5::idesc_bf16(128, 128, 0, 0);
      const uint32_t idesc_acc = tc5::idesc_bf16(128, 128, 0, 1);
      auto issue_st = [&](int t) -> bool {    // S^T = K Q_t^T
        const int st = t % NSQ;
        if (t > 0 && !tc5::mbar_wait(bar(B_SE), (uint32_t)(t - 1) & 1u, abort_flag, p.status, kStatusBit)) return false;
        if (!tc5::mbar_wait(bar(B_QF + st), (uint32_t)(t / NSQ) & 1u, abort_flag, p.status, kStatusBit)) return false;
        tc5::fence_after_sync();
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
          const uint32_t off = (uint32_t)(kk >> 2) * PANEL + (uint32_t)(kk & 3) * 32u;
          tc5::mma_f16(tmem_base + TM_ST, tc5::smem_desc_k_sw128(base + OFF_K + off), tc5::smem_desc_k_sw128(base + OFF_Q + st * TILE + off),
                       idesc_s, kk ? 1u : 0u);
        }
        tc5::mma_commit(bar(B_SF));
        return true;
      };
      auto issue_dpt = [&](int t) {    // dP^T = V dO_t^T (the stage was waited for by issue_st(t))
        const int st = t % NSQ;
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
          const uint32_t off = (uint32_t)(kk >> 2) * PANEL + (uint32_t)(kk & 3) * 32u;
          tc5::mma_f16(tmem_base + TM_DPT, tc5::smem_desc_k_sw128(base + OFF_V + off), tc5::smem_desc_k_sw128(base + OFF_DO + st * TILE + off),
                       idesc_s, kk ? 1u : 0u);
        }
        tc5::mma_commit(bar(B_DF));
      };
      do {
        TC_WAIT(bar(B_KV), 0u);
        if (!issue_st(0)) break;
        issue_dpt(0);
        bool ok = true;
        for (int t = 0; t < n_q; ++t) {
          const int st = t % NSQ;
          // the scores of the next tile go first when their operands are already there (the usual case); otherwise they
          // follow dK of this tile, so that a late Q / dO stage does not hold up the products that are ready
          bool pending = t + 1 < n_q;
          if (pending && tc5::mbar_test(bar(B_SE), (uint32_t)t & 1u) &&
              tc5::mbar_test(bar(B_QF + (t + 1) % NSQ), (uint32_t)((t + 1) / NSQ) & 1u)) {
            if (!issue_st(t + 1)) { ok = false; break; }
            pending = false;
          }
          if (!tc5::mbar_wait(bar(B_PF), (uint32_t)t & 1u, abort_flag, p.status, kStatusBit)) { ok = false; break; }
          tc5::fence_after_sync();
          // dV += P^T dO_t : A = P^T from shared memory (K-major over the 128 queries), B = dO read MN-major
#pragma unroll
          for (int kk = 0; kk < 8; ++kk) {
            tc5::mma_f16(tmem_base + TM_DV, tc5::smem_desc_k_sw128(base + OFF_PT + (uint32_t)(kk >> 2) * PANEL + (uint32_t)(kk & 3) * 32u),
                         tc5::smem_desc_mn_sw128(base + OFF_DO + st * TILE + (uint32_t)kk * 2048u, PANEL), idesc_acc, (t | kk) ? 1u : 0u);
          }
          tc5::mma_commit(bar(B_PE));
          // dK += dS^T Q_t : A = dS^T from tensor memory (group g: 32 packed columns at the start of its half), B = Q MN-major
#pragma unroll
          for (int kk = 0; kk < 8; ++kk) {
            tc5::mma_f16_ta(tmem_base + TM_DK, tmem_base + TM_DPT + (uint32_t)(kk >> 2) * 64u + (uint32_t)(kk & 3) * 8u,
                            tc5::smem_desc_mn_sw128(base + OFF_Q + st * TILE + (uint32_t)kk * 2048u, PANEL), idesc_acc, (t | kk) ? 1u : 0u);
          }
          tc5::mma_commit(bar(B_QE + st));
          if (pending && !issue_st(t + 1)) { ok = false; break; }
          if (t + 1 < n_q) issue_dpt(t + 1);
        }
        if (ok) tc5::mma_commit(bar(B_ACC));
      } while (false);
    }
  } else {
    // ------------------------------------------------------------------ one thread per key row and query half
    const int qd = warp & 3;
    const int wg = (warp - 2) >> 2;    // group g: queries 64 g .. 64 g + 63 of every tile
    const int row = qd * 32 + lane;
    const int grow = k0 + row;
    const uint32_t tlane = tmem_base + ((uint32_t)(qd * 32) << 16);
    const float sl = p.scale * kLog2e;
    const uint32_t prow = base + OFF_PT + (uint32_t)wg * PANEL + (uint32_t)row * 128u;
    const uint32_t swz = (uint32_t)(row & 7);
    bool ok = true;
    for (int t = 0; t < n_q; ++t) {
      const int st = t % NSQ;
      const int qrow0 = (t_first + t) * 128 + wg * 64;    // first query of this group's half
      if (!wait_warp(bar(B_QF + st), (uint32_t)(t / NSQ) & 1u)) { ok = false; break; }
      if (!wait_warp(bar(B_SF), (uint32_t)t & 1u)) { ok = false; break; }
      tc5::fence_after_sync();
      const bool need_mask = p.causal && (qrow0 < k0 + 128);
      const float4* lse2 = reinterpret_cast<const float4*>(s_lse + st * 128 + wg * 64);
      const float4* dlt = reinterpret_cast<const float4*>(s_delta + st * 128 + wg * 64);
      uint32_t rs[2][32], rd[2][32];
      tc5::tmem_ld32(tlane + TM_ST + (uint32_t)wg * 64u, rs[0]);
      tc5::tmem_ld32(tlane + TM_ST + (uint32_t)wg * 64u + 32u, rs[1]);
      tc5::tmem_ld_wait();
      tc5::fence_before_sync();
      __syncwarp();
      if (lane == 0) tc5::mbar_arrive(bar(B_SE));    // the score tile may take tile t + 1
      if (!wait_warp(bar(B_DF), (uint32_t)t & 1u)) { ok = false; break; }
      tc5::fence_after_sync();
      tc5::tmem_ld32(tlane + TM_DPT + (uint32_t)wg * 64u, rd[0]);
      tc5::tmem_ld32(tlane + TM_DPT + (uint32_t)wg * 64u + 32u, rd[1]);
      tc5::tmem_ld_wait();
      if (t > 0 && !wait_warp(bar(B_PE), (uint32_t)(t - 1) & 1u)) { ok = false; break; }    // dV of the previous tile has read P^T
      uint32_t pk[32];
#pragma unroll
      for (int g = 0; g < 8; ++g) {    // 16-byte chunk g = queries 8g .. 8g+7 of this half
        float e[8], ds[8];
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
          const float4 l4 = lse2[g * 2 + hh];
          const float4 d4 = dlt[g * 2 + hh];
          const float la[4] = {l4.x, l4.y, l4.z, l4.w};
          const float da[4] = {d4.x, d4.y, d4.z, d4.w};
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int i = hh * 4 + u;
            const int ql = g * 8 + i;
            float ev = ex2(fmaf(__uint_as_float(rs[ql >> 5][ql & 31]), sl, -la[u]));
            if (need_mask && qrow0 + ql < grow) ev = 0.0f;
            e[i] = ev;
            ds[i] = ev * (__uint_as_float(rd[ql >> 5][ql & 31]) - da[u]);
          }
        }
        st_shared_v4(prow + ((((uint32_t)g) ^ swz) << 4), pack_bf16(e[0], e[1]), pack_bf16(e[2], e[3]), pack_bf16(e[4], e[5]),
                     pack_bf16(e[6], e[7]));
        pk[4 * g] = pack_bf16(ds[0], ds[1]);
        pk[4 * g + 1] = pack_bf16(ds[2], ds[3]);
        pk[4 * g + 2] = pack_bf16(ds[4], ds[5]);
        pk[4 * g + 3] = pack_bf16(ds[6], ds[7]);
      }
      tc5::tmem_st32(tlane + TM_DPT + (uint32_t)wg * 64u, pk);
      tc5::tmem_st_wait();
      tc5::fence_before_sync();
      fence_async_smem();
      __syncwarp();
      if (lane == 0) {
        tc5::mbar_arrive(bar(B_PF));
        tc5::mbar_arrive(bar(B_QE + st));
      }
    }
    if (ok && wait_warp(bar(B_ACC), 0u)) {
      tc5::fence_after_sync();
      __nv_bfloat16* dv = p.dv + (int64_t)b * p.dv_sb + (int64_t)grow * p.dv_ss + (int64_t)h * p.dv_sh;
      __nv_bfloat16* dk = p.dk + (int64_t)b * p.dk_sb + (int64_t)grow * p.dk_ss + (int64_t)h * p.dk_sh;
      // group 0 stores dV, group 1 stores dK
      __nv_bfloat16* dst = wg == 0 ? dv : dk;
      const float f = wg == 0 ? 1.0f : p.scale;
      const uint32_t tsrc = tlane + (wg == 0 ? TM_DV : TM_DK);
#pragma unroll
      for (int c = 0; c < 4; c += 2) {
        uint32_t r0[32], r1[32];
        float v[32];
        tc5::tmem_ld32(tsrc + (uint32_t)c * 32u, r0);
        tc5::tmem_ld32(tsrc + (uint32_t)c * 32u + 32u, r1);
        tc5::tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r0[i]) * f;
        if (grow < p.seqlen) st_row32(dst + c * 32, v);
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r1[i]) * f;
        if (grow < p.seqlen) st_row32(dst + c * 32 + 32, v);
      }
    }
  }

  __syncwarp();
  if (*abort_flag) __nanosleep(200000);
  tc5::fence_before_sync();
  __syncthreads();
  tc5::fence_after_sync();
  if (warp == 1) tc5::tmem_dealloc(tmem_base, TM_COLS);
}

// ================================================================================ dQ, 128-key tiles, dS in tensor memory
namespace dqk2 {
constexpr uint32_t PANEL = 128 * 128;      // [128 rows][64 bf16]: one 64-wide slice of the head dimension
constexpr uint32_t TILE = 2 * PANEL;       // 32 KB: 128 rows x 128 bf16
constexpr int NK = 3;    // K tiles: read by the first (S) and by the last (dQ) MMA of their step, so three are alive
constexpr int NV = 2;    // V tiles: read by dP only
constexpr uint32_t OFF_Q = 0, OFF_DO = TILE, OFF_K = 2 * TILE, OFF_V = OFF_K + NK * TILE, OFF_BAR = OFF_V + NV * TILE;
enum { B_Q = 0, B_KF = 1, B_KE = B_KF + NK, B_VF = B_KE + NK, B_VE = B_VF + NV, B_SF = B_VE + NV, B_SE = B_SF + 1, B_DF = B_SE + 1,
       B_PF = B_DF + 2, B_ACC = B_PF + 2, NBAR = B_ACC + 1 };
constexpr int SMEM = OFF_BAR + NBAR * 8 + 16 + 1024;
// one 128-column score tile, two 128-column dP tiles (dS is written over the dP tile it came from), dQ
constexpr uint32_t TM_S = 0, TM_DP = 128, TM_DQ = 384, TM_COLS = 512;
}    // namespace dqk2

// dQ for 128 query rows; key tiles of 128 (an M = 128 bf16 MMA costs the same ~70 cycles for N = 64 and N = 128, so the
// two score products S = Q K^T and dP = dO V^T are issued over 128 keys at a time).  The eight softmax warps split every
// tile by columns (group g: keys [128 T + 64 g, + 64)).  S is read into registers and its tile released at once; dS is
// packed to bf16 and stored with tcgen05.st over the dP columns it was computed from (group g: the first 32 columns of
// its 64-column half), from where dQ += dS K reads it as the A operand: no shared-memory round trip, and the two dP tiles
// alternate so that dP of tile T + 1 is computed while dS of tile T is still being consumed.  The tensor pipe executes
// MMAs in issue order, so dP(T + 2) may overwrite tile T & 1 once it is issued after dQ(T).
__global__ void __launch_bounds__(kTcThreads, 1)
attn_bwd_dq_tm_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                      const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_do, const TcParams p) {
  using namespace dqk2;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = tc5::smem_u32(smem_raw);
  const uint32_t base = (raw_addr + 1023u) & ~1023u;
  uint8_t* smem = smem_raw + (base - raw_addr);
  const uint32_t bars = base + OFF_BAR;
  auto bar = [&](int i) { return bars + 8u * (uint32_t)i; };
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(smem + OFF_BAR + NBAR * 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);
  auto wait_warp = [&](uint32_t br, uint32_t ph) {
    return __all_sync(0xffffffffu, tc5::mbar_wait(br, ph, abort_flag, p.status, kStatusBit)) != 0;
  };

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int qt = (int)gridDim.x - 1 - (int)blockIdx.x;
  const int bh = blockIdx.y;
  const int b = bh / p.heads;
  const int h = bh - b * p.heads;
  const int q0 = qt * 128;
  const int nk_all = (p.seqlen + 63) / 64;
  const int n_kv = p.causal ? min(2 * qt + 2, nk_all) : nk_all;    // 64-key halves with a visible key
  const int n_t = (n_kv + 1) >> 1;                                 // 128-key tiles; a trailing odd half is fully masked

  if (threadIdx.x == 0) {
    tc5::mbar_init(bar(B_Q), 1);
    for (int s = 0; s < NK; ++s) {
      tc5::mbar_init(bar(B_KF + s), 1);
      tc5::mbar_init(bar(B_KE + s), 1);
    }
    for (int s = 0; s < NV; ++s) {
      tc5::mbar_init(bar(B_VF + s), 1);
      tc5::mbar_init(bar(B_VE + s), 1);
    }
    tc5::mbar_init(bar(B_SF), 1);
    tc5::mbar_init(bar(B_SE), 8);
    for (int s = 0; s < 2; ++s) {
      tc5::mbar_init(bar(B_DF + s), 1);
      tc5::mbar_init(bar(B_PF + s), 8);
    }
    tc5::mbar_init(bar(B_ACC), 1);
    *abort_flag = 0;
    tc5::mbar_fence_init();
    tc5::tma_prefetch_desc(&map_q);
    tc5::tma_prefetch_desc(&map_k);
    tc5::tma_prefetch_desc(&map_v);
    tc5::tma_prefetch_desc(&map_do);
  }
  if (warp == 1) {
    tc5::tmem_alloc(tc5::smem_u32(tmem_holder), TM_COLS);
    tc5::tmem_relinquish();
  }
  tc5::fence_before_sync();
  __syncthreads();
  tc5::fence_after_sync();
  const uint32_t tmem_base = *tmem_holder;

  if (warp == 0) {
    if (lane == 0) {
      tc5::mbar_arrive_expect_tx(bar(B_Q), 2 * TILE);
      tc5::tma_load_4d(base + OFF_Q, &map_q, 0, h, q0, b, bar(B_Q));
      tc5::tma_load_4d(base + OFF_Q + PANEL, &map_q, 64, h, q0, b, bar(B_Q));
      tc5::tma_load_4d(base + OFF_DO, &map_do, 0, h, q0, b, bar(B_Q));
      tc5::tma_load_4d(base + OFF_DO + PANEL, &map_do, 64, h, q0, b, bar(B_Q));
      for (int t = 0; t < n_t; ++t) {
        const int ks = t % NK, vs = t % NV;
        TC_WAIT(bar(B_KE + ks), ((uint32_t)(t / NK) & 1u) ^ 1u);
        tc5::mbar_arrive_expect_tx(bar(B_KF + ks), TILE);
        tc5::tma_load_4d(base + OFF_K + ks * TILE, &map_k, 0, h, t * 128, b, bar(B_KF + ks));
        tc5::tma_load_4d(base + OFF_K + ks * TILE + PANEL, &map_k, 64, h, t * 128, b, bar(B_KF + ks));
        TC_WAIT(bar(B_VE + vs), ((uint32_t)(t / NV) & 1u) ^ 1u);
        tc5::mbar_arrive_expect_tx(bar(B_VF + vs), TILE);
        tc5::tma_load_4d(base + OFF_V + vs * TILE, &map_v, 0, h, t * 128, b, bar(B_VF + vs));
        tc5::tma_load_4d(base + OFF_V + vs * TILE + PANEL, &map_v, 64, h, t * 128, b, bar(B_VF + vs));
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      const uint32_t idesc_s = tc5::idesc_bf16(128, 128, 0, 0);
      const uint32_t idesc_acc = tc5::idesc_bf16(128, 128, 0, 1);
      // S = Q K_t^T (single tile, released by the softmax warps as soon as they hold it in registers) and
      // dP[t & 1] = dO V_t^T
      auto issue_s = [&](int t) -> bool {
        const int ks = t % NK, vs = t % NV;
        if (t > 0 && !tc5::mbar_wait(bar(B_SE), (uint32_t)(t - 1) & 1u, abort_flag, p.status, kStatusBit)) return false;
        if (!tc5::mbar_wait(bar(B_KF + ks), (uint32_t)(t / NK) & 1u, abort_flag, p.status, kStatusBit)) return false;
        tc5::fence_after_sync();
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
          const uint32_t off = (uint32_t)(kk >> 2) * PANEL + (uint32_t)(kk & 3) * 32u;
          tc5::mma_f16(tmem_base + TM_S, tc5::smem_desc_k_sw128(base + OFF_Q + off), tc5::smem_desc_k_sw128(base + OFF_K + ks * TILE + off),
                       idesc_s, kk ? 1u : 0u);
        }
        tc5::mma_commit(bar(B_SF));
        if (!tc5::mbar_wait(bar(B_VF + vs), (uint32_t)(t / NV) & 1u, abort_flag, p.status, kStatusBit)) return false;
        tc5::fence_after_sync();
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
          const uint32_t off = (uint32_t)(kk >> 2) * PANEL + (uint32_t)(kk & 3) * 32u;
          tc5::mma_f16(tmem_base + TM_DP + (uint32_t)(t & 1) * 128u, tc5::smem_desc_k_sw128(base + OFF_DO + off),
                       tc5::smem_desc_k_sw128(base + OFF_V + vs * TILE + off), idesc_s, kk ? 1u : 0u);
        }
        tc5::mma_commit(bar(B_VE + vs));
        tc5::mma_commit(bar(B_DF + (t & 1)));
        return true;
      };
      do {
        TC_WAIT(bar(B_Q), 0u);
        if (!issue_s(0)) break;
        bool ok = true;
        for (int t = 0; t < n_t; ++t) {
          if (t + 1 < n_t && !issue_s(t + 1)) { ok = false; break; }
          const int ks = t % NK;
          if (!tc5::mbar_wait(bar(B_PF + (t & 1)), (uint32_t)(t >> 1) & 1u, abort_flag, p.status, kStatusBit)) { ok = false; break; }
          tc5::fence_after_sync();
          // dQ += dS K_t : A = dS from tensor memory (group g wrote keys 64 g .. 64 g + 63 as 32 packed columns at the start
          // of its half), B = the K tile with the key index as rows (MN-major)
#pragma unroll
          for (int kk = 0; kk < 8; ++kk) {
            tc5::mma_f16_ta(tmem_base + TM_DQ,
                            tmem_base + TM_DP + (uint32_t)(t & 1) * 128u + (uint32_t)(kk >> 2) * 64u + (uint32_t)(kk & 3) * 8u,
                            tc5::smem_desc_mn_sw128(base + OFF_K + ks * TILE + (uint32_t)kk * 2048u, PANEL), idesc_acc, (t | kk) ? 1u : 0u);
          }
          tc5::mma_commit(bar(B_KE + ks));
        }
        if (ok) tc5::mma_commit(bar(B_ACC));
      } while (false);
    }
  } else {
    const int qd = warp & 3;
    const int wg = (warp - 2) >> 2;    // group g: the g-th 64-key half of every tile
    const int row = qd * 32 + lane;
    const int grow = q0 + row;
    const uint32_t tlane = tmem_base + ((uint32_t)(qd * 32) << 16);
    const float sl = p.scale * kLog2e;
    const bool in = grow < p.seqlen;
    const float lse2 = in ? p.lse[(int64_t)bh * p.seqlen + grow] * kLog2e : INFINITY;
    const float dlt = in ? p.delta[(int64_t)bh * p.seqlen + grow] : 0.0f;
    const int lim = p.causal ? min(grow, p.seqlen - 1) : p.seqlen - 1;
    bool ok = true;
    for (int t = 0; t < n_t; ++t) {
      const int col0 = (2 * t + wg) * 64;
      const uint32_t tdp = tlane + TM_DP + (uint32_t)(t & 1) * 128u + (uint32_t)wg * 64u;
      if (!wait_warp(bar(B_SF), (uint32_t)t & 1u)) { ok = false; break; }
      tc5::fence_after_sync();
      const bool need_mask = (p.causal && col0 + 63 > q0) || (col0 + 64 > p.seqlen);
      uint32_t rs[2][32], rd[2][32];
      tc5::tmem_ld32(tlane + TM_S + (uint32_t)wg * 64u, rs[0]);
      tc5::tmem_ld32(tlane + TM_S + (uint32_t)wg * 64u + 32u, rs[1]);
      tc5::tmem_ld_wait();
      tc5::fence_before_sync();
      __syncwarp();
      if (lane == 0) tc5::mbar_arrive(bar(B_SE));    // the score tile may take tile t + 1
      if (!wait_warp(bar(B_DF + (t & 1)), (uint32_t)(t >> 1) & 1u)) { ok = false; break; }
      tc5::fence_after_sync();
      tc5::tmem_ld32(tdp, rd[0]);
      tc5::tmem_ld32(tdp + 32u, rd[1]);
      tc5::tmem_ld_wait();
      uint32_t pk[32];
#pragma unroll
      for (int g = 0; g < 8; ++g) {    // keys 8g .. 8g+7 of this half -> packed columns 4g .. 4g+3
        float ds[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int c = g * 8 + i;
          float e = ex2(fmaf(__uint_as_float(rs[c >> 5][c & 31]), sl, -lse2));
          if (need_mask && col0 + c > lim) e = 0.0f;
          ds[i] = e * (__uint_as_float(rd[c >> 5][c & 31]) - dlt);
        }
        pk[4 * g] = pack_bf16(ds[0], ds[1]);
        pk[4 * g + 1] = pack_bf16(ds[2], ds[3]);
        pk[4 * g + 2] = pack_bf16(ds[4], ds[5]);
        pk[4 * g + 3] = pack_bf16(ds[6], ds[7]);
      }
      tc5::tmem_st32(tdp, pk);
      tc5::tmem_st_wait();
      tc5::fence_before_sync();
      __syncwarp();
      if (lane == 0) tc5::mbar_arrive(bar(B_PF + (t & 1)));
    }
    if (ok && wait_warp(bar(B_ACC), 0u)) {
      tc5::fence_after_sync();
      __nv_bfloat16* dq = p.dq + (int64_t)b * p.dq_sb + (int64_t)grow * p.dq_ss + (int64_t)h * p.dq_sh;
      // each group stores one half of the row
      uint32_t r0[32], r1[32];
      float v[32];
      tc5::tmem_ld32(tlane + TM_DQ + (uint32_t)wg * 64u, r0);
      tc5::tmem_ld32(tlane + TM_DQ + (uint32_t)wg * 64u + 32u, r1);
      tc5::tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r0[i]) * p.scale;
      if (in) st_row32(dq + wg * 64, v);
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r1[i]) * p.scale;
      if (in) st_row32(dq + wg * 64 + 32, v);
    }
  }

  __syncwarp();
  if (*abort_flag) __nanosleep(200000);
  tc5::fence_before_sync();
  __syncthreads();
  tc5::fence_after_sync();
  if (warp == 1) tc5::tmem_dealloc(tmem_base, TM_COLS);
}

// ============================================================================ dQ, persistent CTAs over the work items
namespace dqk3 {
using namespace dqk2;
enum { B3_QE = NBAR, B3_OE = NBAR + 1, NBAR3 = NBAR + 2 };
template <int D>
struct Cfg {
  static constexpr int HP = D / 64;
  static constexpr uint32_t TILE = HP * PANEL;    // 128 rows of one head
  static constexpr uint32_t OFF_DO = TILE, OFF_K = 2 * TILE, OFF_V = OFF_K + NK * TILE, OFF_BAR = OFF_V + NV * TILE;
  static constexpr int SMEM = OFF_BAR + NBAR3 * 8 + 16 + 1024;
};
}    // namespace dqk3

// attn_bwd_dq_tm_kernel with one CTA per SM walking the (query tile, batch * head) items, the exponentials taken before dP is
// waited for, the next K and V tile probed while MMAs run, and dQ stored in whole lines: 4 x 2048 x 32 heads of 128, causal,
// 235 -> 206 us.  Rings, the score tile and
// the dP tiles keep running across items (one global tile counter), so Q / dO / K / V of the next item are loaded and
// its first score products issued while the softmax warps still store dQ of the current one.  B3_QE: the score products
// of an item are complete, Q and dO may be overwritten; B3_OE: the softmax warps have read dQ, the accumulator may be
// overwritten by the first product of the next item.
template <int D>
__global__ void __launch_bounds__(kPsThreads, 1)
attn_bwd_dq_ps_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                      const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_do, const TcParams p, int n_qt,
                      int n_items) {
  using namespace dqk3;
  constexpr int HP = Cfg<D>::HP;
  constexpr uint32_t TILE = Cfg<D>::TILE, OFF_DO = Cfg<D>::OFF_DO, OFF_K = Cfg<D>::OFF_K, OFF_V = Cfg<D>::OFF_V, OFF_BAR = Cfg<D>::OFF_BAR;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = tc5::smem_u32(smem_raw);
  const uint32_t base = (raw_addr + 1023u) & ~1023u;
  uint8_t* smem = smem_raw + (base - raw_addr);
  const uint32_t bars = base + OFF_BAR;
  auto bar = [&](int i) { return bars + 8u * (uint32_t)i; };
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(smem + OFF_BAR + NBAR3 * 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);
  auto wait_warp = [&](uint32_t br, uint32_t ph) {
    return __all_sync(0xffffffffu, tc5::mbar_wait(br, ph, abort_flag, p.status, kStatusBit)) != 0;
  };
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int nk_all = (p.seqlen + 63) / 64;
  const ItemOrder order{n_qt, p.batch * p.heads, p.group};
  const int n_waves = (n_items + (int)gridDim.x - 1) / (int)gridDim.x;
  auto item_at = [&](int w) {
    const int c = (w & 1) ? (int)gridDim.x - 1 - (int)blockIdx.x : (int)blockIdx.x;
    return w * (int)gridDim.x + c;
  };
  auto tiles_of = [&](int qt) {
    const int n_kv = p.causal ? min(2 * qt + 2, nk_all) : nk_all;
    return (n_kv + 1) >> 1;
  };

  if (threadIdx.x == 0) {
    tc5::mbar_init(bar(B_Q), 1);
    for (int s = 0; s < NK; ++s) {
      tc5::mbar_init(bar(B_KF + s), 1);
      tc5::mbar_init(bar(B_KE + s), 1);
    }
    for (int s = 0; s < NV; ++s) {
      tc5::mbar_init(bar(B_VF + s), 1);
      tc5::mbar_init(bar(B_VE + s), 1);
    }
    tc5::mbar_init(bar(B_SF), 1);
    tc5::mbar_init(bar(B_SE), 8);
    for (int s = 0; s < 2; ++s) {
      tc5::mbar_init(bar(B_DF + s), 1);
      tc5::mbar_init(bar(B_PF + s), 8);
    }
    tc5::mbar_init(bar(B_ACC), 1);
    tc5::mbar_init(bar(B3_QE), 1);
    tc5::mbar_init(bar(B3_OE), 8);
    *abort_flag = 0;
    tc5::mbar_fence_init();
    tc5::tma_prefetch_desc(&map_q);
    tc5::tma_prefetch_desc(&map_k);
    tc5::tma_prefetch_desc(&map_v);
    tc5::tma_prefetch_desc(&map_do);
  }
  if (warp == 1) {
    tc5::tmem_alloc(tc5::smem_u32(tmem_holder), TM_COLS);
    tc5::tmem_relinquish();
  }
  tc5::fence_before_sync();
  __syncthreads();
  tc5::fence_after_sync();
  const uint32_t tmem_base = *tmem_holder;

  if (warp < 4) {
    regs_aux<88>();
    if (warp == 0 && lane == 0) {
      int gt = 0, it = 0;
      bool ok = true;
      for (int w = 0; w < n_waves && ok; ++w) {
        const int item = item_at(w);
        if (item >= n_items) continue;
        int level, bh;
        order.decode(item, level, bh);
        const int qt = n_qt - 1 - level;
        const int b = bh / p.heads, h = bh - b * p.heads;
        const int n_t = tiles_of(qt);
        if (it > 0 && !tc5::mbar_wait(bar(B3_QE), (uint32_t)(it - 1) & 1u, abort_flag, p.status, kStatusBit)) break;
        tc5::mbar_arrive_expect_tx(bar(B_Q), 2 * TILE);
#pragma unroll
        for (int pp = 0; pp < HP; ++pp) {
          tc5::tma_load_4d(base + OFF_Q + pp * PANEL, &map_q, pp * 64, h, qt * 128, b, bar(B_Q));
          tc5::tma_load_4d(base + OFF_DO + pp * PANEL, &map_do, pp * 64, h, qt * 128, b, bar(B_Q));
        }
        for (int t = 0; t < n_t; ++t, ++gt) {
          const int ks = gt % NK, vs = gt % NV;
          if (!tc5::mbar_wait(bar(B_KE + ks), ((uint32_t)(gt / NK) & 1u) ^ 1u, abort_flag, p.status, kStatusBit)) { ok = false; break; }
          tc5::mbar_arrive_expect_tx(bar(B_KF + ks), TILE);
#pragma unroll
          for (int pp = 0; pp < HP; ++pp) tc5::tma_load_4d(base + OFF_K + ks * TILE + pp * PANEL, &map_k, pp * 64, h, t * 128, b, bar(B_KF + ks));
          if (!tc5::mbar_wait(bar(B_VE + vs), ((uint32_t)(gt / NV) & 1u) ^ 1u, abort_flag, p.status, kStatusBit)) { ok = false; break; }
          tc5::mbar_arrive_expect_tx(bar(B_VF + vs), TILE);
#pragma unroll
          for (int pp = 0; pp < HP; ++pp) tc5::tma_load_4d(base + OFF_V + vs * TILE + pp * PANEL, &map_v, pp * 64, h, t * 128, b, bar(B_VF + vs));
        }
        ++it;
      }
    } else if (warp == 1 && lane == 0) {
      const uint32_t idesc_s = tc5::idesc_bf16(128, 128, 0, 0);
      const uint32_t idesc_acc = tc5::idesc_bf16(128, D, 0, 1);
      Ring<NK> kr, kq;    // K tile of the next score product, of the next dQ product
      Ring<NV> vr;
      bool k_ready = false, v_ready = false;    // probes of the next K and V tile, made while MMAs were running
      // S = Q K^T and dP[gt & 1] = dO V^T for the gt-th tile of this CTA
      auto issue_s = [&](int gt) -> bool {
        const int ks = kr.slot, vs = vr.slot;
        // data barriers first (they pass while the softmax warps still hold S), so that the two products are issued back
        // to back once S is free: a wait between them idles the tensor pipe for 100+ cycles even when V is there
        if (!k_ready && !tc5::mbar_wait(bar(B_KF + ks), kr.phase, abort_flag, p.status, kStatusBit)) return false;
        if (!v_ready && !tc5::mbar_wait(bar(B_VF + vs), vr.phase, abort_flag, p.status, kStatusBit)) return false;
        if (gt > 0 && !tc5::mbar_wait(bar(B_SE), (uint32_t)(gt - 1) & 1u, abort_flag, p.status, kStatusBit)) return false;
        tc5::fence_after_sync();
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          const uint32_t off = (uint32_t)(kk >> 2) * PANEL + (uint32_t)(kk & 3) * 32u;
          tc5::mma_f16(tmem_base + TM_S, tc5::smem_desc_k_sw128(base + OFF_Q + off), tc5::smem_desc_k_sw128(base + OFF_K + ks * TILE + off),
                       idesc_s, kk ? 1u : 0u);
        }
        tc5::mma_commit(bar(B_SF));
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          const uint32_t off = (uint32_t)(kk >> 2) * PANEL + (uint32_t)(kk & 3) * 32u;
          tc5::mma_f16(tmem_base + TM_DP + (uint32_t)(gt & 1) * 128u, tc5::smem_desc_k_sw128(base + OFF_DO + off),
                       tc5::smem_desc_k_sw128(base + OFF_V + vs * TILE + off), idesc_s, kk ? 1u : 0u);
        }
        tc5::mma_commit(bar(B_VE + vs));
        tc5::mma_commit(bar(B_DF + (gt & 1)));
        kr.next();
        vr.next();
        k_ready = tc5::mbar_test(bar(B_KF + kr.slot), kr.phase);
        v_ready = tc5::mbar_test(bar(B_VF + vr.slot), vr.phase);
        return true;
      };
      int g0 = 0, it = 0;
      bool ok = true;
      for (int w = 0; w < n_waves && ok; ++w) {
        const int item = item_at(w);
        if (item >= n_items) continue;
        int level, bh;
        order.decode(item, level, bh);
        const int n_t = tiles_of(n_qt - 1 - level);
        if (!tc5::mbar_wait(bar(B_Q), (uint32_t)it & 1u, abort_flag, p.status, kStatusBit)) { ok = false; break; }
        if (!issue_s(g0)) { ok = false; break; }
        if (n_t == 1) tc5::mma_commit(bar(B3_QE));
        if (it > 0 && !tc5::mbar_wait(bar(B3_OE), (uint32_t)(it - 1) & 1u, abort_flag, p.status, kStatusBit)) { ok = false; break; }
        for (int t = 0; t < n_t; ++t) {
          const int gt = g0 + t;
          if (t + 1 < n_t) {
            if (!issue_s(gt + 1)) { ok = false; break; }
            if (t + 2 == n_t) tc5::mma_commit(bar(B3_QE));    // every score product of this item is issued
          }
          const int ks = kq.slot;
          kq.next();
          if (!tc5::mbar_wait(bar(B_PF + (gt & 1)), (uint32_t)(gt >> 1) & 1u, abort_flag, p.status, kStatusBit)) { ok = false; break; }
          tc5::fence_after_sync();
#pragma unroll
          for (int kk = 0; kk < 8; ++kk) {
            tc5::mma_f16_ta(tmem_base + TM_DQ,
                            tmem_base + TM_DP + (uint32_t)(gt & 1) * 128u + (uint32_t)(kk >> 2) * 64u + (uint32_t)(kk & 3) * 8u,
                            tc5::smem_desc_mn_sw128(base + OFF_K + ks * TILE + (uint32_t)kk * 2048u, PANEL), idesc_acc, (t | kk) ? 1u : 0u);
          }
          tc5::mma_commit(bar(B_KE + ks));
        }
        if (!ok) break;
        tc5::mma_commit(bar(B_ACC));
        g0 += n_t;
        ++it;
      }
    }
  } else {
    regs_softmax<88>();
    const int qd = warp & 3;
    const int wg = (warp - 4) >> 2;    // group g: the g-th 64-key half of every tile
    const int row = qd * 32 + lane;
    const uint32_t tlane = tmem_base + ((uint32_t)(qd * 32) << 16);
    const float sl = p.scale * kLog2e;
    int g0 = 0, it = 0;
    bool ok = true;
    for (int w = 0; w < n_waves && ok; ++w) {
      const int item = item_at(w);
      if (item >= n_items) continue;
      int level, bh;
      order.decode(item, level, bh);
      const int qt = n_qt - 1 - level;
      const int b = bh / p.heads, h = bh - b * p.heads;
      const int n_t = tiles_of(qt);
      const int q0 = qt * 128;
      const int grow = q0 + row;
      const bool in = grow < p.seqlen;
      const float lse2 = in ? p.lse[(int64_t)bh * p.seqlen + grow] * kLog2e : INFINITY;
      const float dlt = in ? p.delta[(int64_t)bh * p.seqlen + grow] : 0.0f;
      const uint64_t sl2 = f2_pack(sl, sl), nlse2 = f2_pack(-lse2, -lse2), ndlt2 = f2_pack(-dlt, -dlt);
      const int lim = p.causal ? min(grow, p.seqlen - 1) : p.seqlen - 1;
      for (int t = 0; t < n_t; ++t) {
        const int gt = g0 + t;
        const int col0 = (2 * t + wg) * 64;
        const uint32_t tdp = tlane + TM_DP + (uint32_t)(gt & 1) * 128u + (uint32_t)wg * 64u;
        if (!wait_warp(bar(B_SF), (uint32_t)gt & 1u)) { ok = false; break; }
        tc5::fence_after_sync();
        const bool need_mask = (p.causal && col0 + 63 > q0) || (col0 + 64 > p.seqlen);
        uint32_t rs[2][32], rd[2][32];    // the scores become probabilities while dP is still being computed
        tc5::tmem_ld32(tlane + TM_S + (uint32_t)wg * 64u, rs[0]);
        tc5::tmem_ld32(tlane + TM_S + (uint32_t)wg * 64u + 32u, rs[1]);
        tc5::tmem_ld_wait();
        tc5::fence_before_sync();
        __syncwarp();
        if (lane == 0) tc5::mbar_arrive(bar(B_SE));    // the score tile may take the next tile
        // dS = exp2(s * sl - lse) * (dP - delta), two columns per instruction
#pragma unroll
        for (int i = 0; i < 64; i += 2) {
          uint32_t &r0 = rs[i >> 5][i & 31], &r1 = rs[i >> 5][(i & 31) + 1];
          const float2 x = f2_unpack(f2_fma(f2_pack(__uint_as_float(r0), __uint_as_float(r1)), sl2, nlse2));
          r0 = __float_as_uint(ex2(x.x));
          r1 = __float_as_uint(ex2(x.y));
        }
        if (need_mask) mask_above(rs, lim - col0, 0u);
        if (!wait_warp(bar(B_DF + (gt & 1)), (uint32_t)(gt >> 1) & 1u)) { ok = false; break; }
        tc5::fence_after_sync();
        tc5::tmem_ld32(tdp, rd[0]);
        tc5::tmem_ld32(tdp + 32u, rd[1]);
        tc5::tmem_ld_wait();
        uint32_t pk[32];
#pragma unroll
        for (int i = 0; i < 64; i += 2) {
          const uint64_t e = f2_pack(__uint_as_float(rs[i >> 5][i & 31]), __uint_as_float(rs[i >> 5][(i & 31) + 1]));
          const uint64_t d = f2_pack(__uint_as_float(rd[i >> 5][i & 31]), __uint_as_float(rd[i >> 5][(i & 31) + 1]));
          const float2 ds = f2_unpack(f2_mul(e, f2_add(d, ndlt2)));
          pk[i >> 1] = pack_bf16(ds.x, ds.y);
        }
        tc5::tmem_st32(tdp, pk);
        tc5::tmem_st_wait();
        tc5::fence_before_sync();
        __syncwarp();
        if (lane == 0) tc5::mbar_arrive(bar(B_PF + (gt & 1)));
      }
      if (!ok || !wait_warp(bar(B_ACC), (uint32_t)it & 1u)) { ok = false; break; }
      tc5::fence_after_sync();
      // 64 columns per group; of a head of 64, group 0 stores all and group 1 nothing
      __nv_bfloat16* dq = p.dq + (int64_t)b * p.dq_sb + (int64_t)(q0 + qd * 32) * p.dq_ss + (int64_t)h * p.dq_sh;
      const bool mine = wg < HP;
      uint32_t r[2][32];
      if (mine) {
        tc5::tmem_ld32(tlane + TM_DQ + (uint32_t)wg * 64u, r[0]);
        tc5::tmem_ld32(tlane + TM_DQ + (uint32_t)wg * 64u + 32u, r[1]);
        tc5::tmem_ld_wait();
      }
      tc5::fence_before_sync();
      __syncwarp();
      if (lane == 0) tc5::mbar_arrive(bar(B3_OE));    // the accumulator may take the next item
      if (mine) {
        float v[64];
#pragma unroll
        for (int i = 0; i < 64; ++i) v[i] = __uint_as_float(r[i >> 5][i & 31]) * p.scale;
        st_rows64(dq + wg * 64, p.dq_ss, p.seqlen - q0 - qd * 32, v);
      }
      g0 += n_t;
      ++it;
    }
  }

  __syncwarp();
  if (*abort_flag) __nanosleep(200000);
  tc5::fence_before_sync();
  __syncthreads();
  tc5::fence_after_sync();
  if (warp == 1) tc5::tmem_dealloc(tmem_base, TM_COLS);
}

// ====================================================================== dK / dV, persistent CTAs over the work items
namespace dkv3 {
// Head size 128 fills tensor memory (S^T, dP^T, dV, dK: 4 x 128 columns).  P^T is therefore written over the scores it came
// from and dS^T over its dP^T, and the tensor pipe takes dV, S^T of the next tile, dK, dP^T of the next tile, in this order
// per tile: each overwrites what the product before it has read.  Shared memory then has room for a third Q stage (the scores
// want Q of tile t + 1 while dK still has to read Q of tile t).
// Head size 64 leaves 128 columns and 64 KB free: a second dP^T and P^T in shared memory (two buffers), so that neither the
// score products nor the softmax warps wait for the products of the previous tile.
template <int D>
struct Cfg {
  static constexpr int HP = D / 64;
  static constexpr bool PT_TMEM = D == 128;       // P^T over S^T in tensor memory, else in shared memory
  static constexpr int NQ = 3;                    // Q stages
  static constexpr int ND = D == 128 ? 2 : 3;     // dO stages (with the rows of lse and delta)
  static constexpr int NB = D == 128 ? 1 : 2;     // P^T and dP^T buffers
  static constexpr uint32_t PANEL = 128 * 128, TILE = HP * PANEL, TILE_P = 2 * PANEL;
  static constexpr uint32_t OFF_V = TILE, OFF_Q = 2 * TILE, OFF_DO = OFF_Q + NQ * TILE, OFF_PT = OFF_DO + ND * TILE,
                            OFF_LSE = OFF_PT + (PT_TMEM ? 0 : NB * TILE_P), OFF_BAR = OFF_LSE + ND * 2 * 128 * 4;
  static constexpr int B_KV = 0, B_QF = 1, B_QE = B_QF + NQ, B_OF = B_QE + NQ, B_OE = B_OF + ND, B_SF = B_OE + ND, B_SE = B_SF + 1, B_DF = B_SE + 1,
                       B_PF = B_DF + NB, B_PP = B_PF + NB, B_PE = B_PP + NB, B_ACC = B_PE + NB, B3_KVE = B_ACC + 1, B3_OE = B3_KVE + 1,
                       NBAR = B3_OE + 1;
  static constexpr int SMEM = OFF_BAR + NBAR * 8 + 16;    // head size 128: 848 bytes below the limit, so the base has to be aligned
  static constexpr uint32_t TM_ST = 0, TM_DPT = 128, TM_DV = TM_DPT + NB * 128, TM_DK = TM_DV + D, TM_COLS = 512;
  static_assert(SMEM <= 227 * 1024, "persistent dK/dV kernel: shared memory");
  static_assert(TM_DK + D <= TM_COLS, "persistent dK/dV kernel: tensor memory");
};
}    // namespace dkv3

// dK and dV for 128 key rows, one CTA per SM walking the (key tile, batch * head) items; the Q and dO stages, the score tiles
// and all barriers keep running across items (one global query-tile counter).  The softmax warps hand over P^T as soon as it
// is stored, so that dV runs under the arithmetic of dS^T, and take dP^T only then, so that dK of the previous tile and dP^T
// run under the exponentials.  Bound by the tensor pipe for head size 128 (32 MMAs of 80 to 110 cycles per 128 x 128 tile)
// and by the softmax warps for 64.  4 x 2048 x 32 heads of 128, causal: 398 -> 297 us (waiting for dP^T before any
// exponential, one barrier for P^T and dS^T, and stores of one row per lane before).
// B3_KVE: every S^T / dP^T product of an item is complete, K and V may be overwritten by the next item's; B3_OE: the softmax
// warps have read dV and dK, the first products of the next item may overwrite the accumulators.
template <int D>
__global__ void __launch_bounds__(kPsThreads, 1)
attn_bwd_dkdv_ps_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                        const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_do, const TcParams p, int n_kt,
                        int n_items) {
  using C = dkv3::Cfg<D>;
  constexpr int HP = C::HP, NQ = C::NQ, ND = C::ND, NB = C::NB;
  constexpr bool PT_TMEM = C::PT_TMEM;
  constexpr uint32_t PANEL = C::PANEL, TILE = C::TILE, TILE_P = C::TILE_P, OFF_K = 0, OFF_V = C::OFF_V, OFF_Q = C::OFF_Q, OFF_DO = C::OFF_DO,
                     OFF_PT = C::OFF_PT, OFF_LSE = C::OFF_LSE, OFF_BAR = C::OFF_BAR;
  constexpr int B_KV = C::B_KV, B_QF = C::B_QF, B_QE = C::B_QE, B_OF = C::B_OF, B_OE = C::B_OE, B_SF = C::B_SF, B_SE = C::B_SE, B_DF = C::B_DF, B_PF = C::B_PF, B_PP = C::B_PP, B_PE = C::B_PE,
                B_ACC = C::B_ACC, B3_KVE = C::B3_KVE, B3_OE = C::B3_OE;
  constexpr uint32_t TM_ST = C::TM_ST, TM_DPT = C::TM_DPT, TM_DV = C::TM_DV, TM_DK = C::TM_DK, TM_COLS = C::TM_COLS;
  extern __shared__ __align__(1024) uint8_t smem[];
  const uint32_t base = tc5::smem_u32(smem);
  if ((base & 1023u) != 0u) {    // never seen: the declared alignment is kept
    if (threadIdx.x == 0) atomicOr(p.status, kStatusBit);
    return;
  }
  const uint32_t bars = base + OFF_BAR;
  auto bar = [&](int i) { return bars + 8u * (uint32_t)i; };
  float* s_lse = reinterpret_cast<float*>(smem + OFF_LSE);    // [ND][128] -lse in log2 units, then [ND][128] -delta
  float* s_delta = s_lse + ND * 128;
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(smem + OFF_BAR + C::NBAR * 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);
  auto wait_warp = [&](uint32_t br, uint32_t ph) {
    return __all_sync(0xffffffffu, tc5::mbar_wait(br, ph, abort_flag, p.status, kStatusBit)) != 0;
  };
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int nq_all = (p.seqlen + 127) / 128;
  const ItemOrder order{n_kt, p.batch * p.heads, p.group};
  const int n_waves = (n_items + (int)gridDim.x - 1) / (int)gridDim.x;
  auto item_at = [&](int w) {
    const int c = (w & 1) ? (int)gridDim.x - 1 - (int)blockIdx.x : (int)blockIdx.x;
    return w * (int)gridDim.x + c;
  };

  if (threadIdx.x == 0) {
    tc5::mbar_init(bar(B_KV), 1);
    for (int s = 0; s < NQ; ++s) {
      tc5::mbar_init(bar(B_QF + s), 1);
      tc5::mbar_init(bar(B_QE + s), 1);
    }
    for (int s = 0; s < ND; ++s) {
      tc5::mbar_init(bar(B_OF + s), 2);    // TMA bytes + the lse / delta rows written by warp 0
      tc5::mbar_init(bar(B_OE + s), 9);    // last MMA that reads the stage + eight softmax warps
    }
    tc5::mbar_init(bar(B_SF), 1);
    tc5::mbar_init(bar(B_SE), 8);
    for (int s = 0; s < NB; ++s) {
      tc5::mbar_init(bar(B_DF + s), 1);
      tc5::mbar_init(bar(B_PF + s), 8);    // dS^T stored
      tc5::mbar_init(bar(B_PP + s), 8);    // P^T stored
      tc5::mbar_init(bar(B_PE + s), 1);
    }
    tc5::mbar_init(bar(B_ACC), 1);
    tc5::mbar_init(bar(B3_KVE), 1);
    tc5::mbar_init(bar(B3_OE), 8);
    *abort_flag = 0;
    tc5::mbar_fence_init();
    tc5::tma_prefetch_desc(&map_q);
    tc5::tma_prefetch_desc(&map_k);
    tc5::tma_prefetch_desc(&map_v);
    tc5::tma_prefetch_desc(&map_do);
  }
  if (warp == 1) {
    tc5::tmem_alloc(tc5::smem_u32(tmem_holder), TM_COLS);
    tc5::tmem_relinquish();
  }
  tc5::fence_before_sync();
  __syncthreads();
  tc5::fence_after_sync();
  const uint32_t tmem_base = *tmem_holder;

  if (warp < 4) {
    regs_aux<88>();
    if (warp == 0) {
    // ------------------------------------------------------------------ producer (whole warp: lane 0 issues TMA)
    int gq = 0, it = 0;
    bool ok = true;
    for (int w = 0; w < n_waves && ok; ++w) {
      const int item = item_at(w);
      if (item >= n_items) continue;
      int kt, bh;
      order.decode(item, kt, bh);
      const int b = bh / p.heads, h = bh - b * p.heads;
      const int k0 = kt * 128;
      const int t_first = p.causal ? kt : 0;
      const int n_q = nq_all - t_first;
      if (it > 0 && !__all_sync(0xffffffffu, tc5::mbar_wait(bar(B3_KVE), (uint32_t)(it - 1) & 1u, abort_flag, p.status, kStatusBit))) break;
      if (lane == 0) {
        tc5::mbar_arrive_expect_tx(bar(B_KV), 2 * TILE);
#pragma unroll
        for (int pp = 0; pp < HP; ++pp) {
          tc5::tma_load_4d(base + OFF_K + pp * PANEL, &map_k, pp * 64, h, k0, b, bar(B_KV));
          tc5::tma_load_4d(base + OFF_V + pp * PANEL, &map_v, pp * 64, h, k0, b, bar(B_KV));
        }
      }
      const float* glse = p.lse + (int64_t)bh * p.seqlen;
      const float* gdelta = p.delta + (int64_t)bh * p.seqlen;
      for (int t = 0; t < n_q; ++t, ++gq) {
        const int s = gq % NQ, so = gq % ND;
        const int qrow0 = (t_first + t) * 128;
        if (!__all_sync(0xffffffffu, tc5::mbar_wait(bar(B_QE + s), ((uint32_t)(gq / NQ) & 1u) ^ 1u, abort_flag, p.status, kStatusBit))) { ok = false; break; }
        if (lane == 0) {
          tc5::mbar_arrive_expect_tx(bar(B_QF + s), TILE);
#pragma unroll
          for (int pp = 0; pp < HP; ++pp) tc5::tma_load_4d(base + OFF_Q + s * TILE + pp * PANEL, &map_q, pp * 64, h, qrow0, b, bar(B_QF + s));
        }
        if (!__all_sync(0xffffffffu, tc5::mbar_wait(bar(B_OE + so), ((uint32_t)(gq / ND) & 1u) ^ 1u, abort_flag, p.status, kStatusBit))) { ok = false; break; }
        if (lane == 0) {
          tc5::mbar_arrive_expect_tx(bar(B_OF + so), TILE);
#pragma unroll
          for (int pp = 0; pp < HP; ++pp) tc5::tma_load_4d(base + OFF_DO + so * TILE + pp * PANEL, &map_do, pp * 64, h, qrow0, b, bar(B_OF + so));
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int r = lane + 32 * i;
          const bool in = qrow0 + r < p.seqlen;
          s_lse[so * 128 + r] = in ? -(glse[qrow0 + r] * kLog2e) : -INFINITY;    // -inf makes the probability exactly zero
          s_delta[so * 128 + r] = in ? -gdelta[qrow0 + r] : 0.0f;
        }
        __syncwarp();
        if (lane == 0) tc5::mbar_arrive(bar(B_OF + so));
      }
      ++it;
    }
    } else if (warp == 1 && lane == 0) {
    // ------------------------------------------------------------------ MMA issuer
      const uint32_t idesc_s = tc5::idesc_bf16(128, 128, 0, 0);
      const uint32_t idesc_acc = tc5::idesc_bf16(128, D, 0, 1);
      auto wait_for = [&](int i, int n) { return tc5::mbar_wait(bar(i), (uint32_t)n & 1u, abort_flag, p.status, kStatusBit); };
      // S^T = K Q^T for the gq-th query tile of this CTA; the caller has waited for its Q and for the score tile
      auto issue_st = [&](int gq) {
        const int st = gq % NQ;
        tc5::fence_after_sync();
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          const uint32_t off = (uint32_t)(kk >> 2) * PANEL + (uint32_t)(kk & 3) * 32u;
          tc5::mma_f16(tmem_base + TM_ST, tc5::smem_desc_k_sw128(base + OFF_K + off), tc5::smem_desc_k_sw128(base + OFF_Q + st * TILE + off),
                       idesc_s, kk ? 1u : 0u);
        }
        tc5::mma_commit(bar(B_SF));
      };
      // dP^T = V dO^T.  The tensor pipe executes in issue order: with one buffer this is issued after dK of tile gq - 1, with
      // two after dK of tile gq - 2, so no "buffer free" barrier is needed.
      auto issue_dpt = [&](int gq, bool there) -> bool {    // there: its dO has been probed
        const int so = gq % ND;
        if (!there && !wait_for(B_OF + so, gq / ND)) return false;
        tc5::fence_after_sync();
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          const uint32_t off = (uint32_t)(kk >> 2) * PANEL + (uint32_t)(kk & 3) * 32u;
          tc5::mma_f16(tmem_base + TM_DPT + (uint32_t)(gq % NB) * 128u, tc5::smem_desc_k_sw128(base + OFF_V + off),
                       tc5::smem_desc_k_sw128(base + OFF_DO + so * TILE + off), idesc_s, kk ? 1u : 0u);
        }
        tc5::mma_commit(bar(B_DF + gq % NB));
        return true;
      };
      auto issue_dv = [&](int gq, bool first) {
        const int so = gq % ND;
        tc5::fence_after_sync();
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
          const uint64_t d_o = tc5::smem_desc_mn_sw128(base + OFF_DO + so * TILE + (uint32_t)kk * 2048u, PANEL);
          const uint32_t acc = (!first || kk) ? 1u : 0u;
          if (PT_TMEM)
            tc5::mma_f16_ta(tmem_base + TM_DV, tmem_base + TM_ST + (uint32_t)(kk >> 2) * 64u + (uint32_t)(kk & 3) * 8u, d_o, idesc_acc, acc);
          else
            tc5::mma_f16(tmem_base + TM_DV, tc5::smem_desc_k_sw128(base + OFF_PT + (uint32_t)(gq % NB) * TILE_P + (uint32_t)(kk >> 2) * PANEL + (uint32_t)(kk & 3) * 32u),
                         d_o, idesc_acc, acc);
        }
        tc5::mma_commit(bar(B_OE + so));
        if (!PT_TMEM) tc5::mma_commit(bar(B_PE + gq % NB));
      };
      auto issue_dk = [&](int gq, bool first) {
        const int st = gq % NQ;
        tc5::fence_after_sync();
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
          tc5::mma_f16_ta(tmem_base + TM_DK, tmem_base + TM_DPT + (uint32_t)(gq % NB) * 128u + (uint32_t)(kk >> 2) * 64u + (uint32_t)(kk & 3) * 8u,
                          tc5::smem_desc_mn_sw128(base + OFF_Q + st * TILE + (uint32_t)kk * 2048u, PANEL), idesc_acc, (!first || kk) ? 1u : 0u);
        }
        tc5::mma_commit(bar(B_QE + st));
      };
      int g0 = 0, it = 0;
      bool ok = true;
      for (int w = 0; w < n_waves && ok; ++w) {
        const int item = item_at(w);
        if (item >= n_items) continue;
        int kt, bh;
        order.decode(item, kt, bh);
        const int n_q = nq_all - (p.causal ? kt : 0);
        if (!tc5::mbar_wait(bar(B_KV), (uint32_t)it & 1u, abort_flag, p.status, kStatusBit)) { ok = false; break; }
        if (!wait_for(B_QF + g0 % NQ, g0 / NQ)) { ok = false; break; }
        if (!PT_TMEM && g0 > 0 && !wait_for(B_SE, g0 - 1)) { ok = false; break; }
        issue_st(g0);
        if (!issue_dpt(g0, false)) { ok = false; break; }
        if (n_q == 1) tc5::mma_commit(bar(B3_KVE));
        if (it > 0 && !wait_for(B3_OE, it - 1)) { ok = false; break; }
        for (int t = 0; t < n_q; ++t) {
          const int gq = g0 + t;
          const bool more = t + 1 < n_q;
          if (PT_TMEM) {
            if (!wait_for(B_PP, gq)) { ok = false; break; }
            issue_dv(gq, t == 0);
            if (more) {    // over the P^T that dV reads: in issue order
              if (!wait_for(B_QF + (gq + 1) % NQ, (gq + 1) / NQ)) { ok = false; break; }
              issue_st(gq + 1);
            }
            if (!wait_for(B_PF, gq)) { ok = false; break; }
            issue_dk(gq, t == 0);
            if (more && !issue_dpt(gq + 1, false)) { ok = false; break; }
            if (t + 2 == n_q) tc5::mma_commit(bar(B3_KVE));    // every S^T / dP^T product of this item is issued
          } else {
            // the softmax warps release S^T right after reading it, long before P^T of this tile is there: the scores of the
            // next tile are computed under their exponentials, unless its Q or dO is still on the way
            bool pending = more;
            if (pending && !wait_for(B_SE, gq)) { ok = false; break; }
            if (pending && tc5::mbar_test(bar(B_QF + (gq + 1) % NQ), (uint32_t)((gq + 1) / NQ) & 1u) &&
                tc5::mbar_test(bar(B_OF + (gq + 1) % ND), (uint32_t)((gq + 1) / ND) & 1u)) {
              issue_st(gq + 1);
              issue_dpt(gq + 1, true);
              pending = false;
            }
            if (!wait_for(B_PP + gq % NB, gq / NB)) { ok = false; break; }
            issue_dv(gq, t == 0);
            if (!wait_for(B_PF + gq % NB, gq / NB)) { ok = false; break; }
            issue_dk(gq, t == 0);
            if (pending) {
              if (!wait_for(B_QF + (gq + 1) % NQ, (gq + 1) / NQ)) { ok = false; break; }
              issue_st(gq + 1);
              if (!issue_dpt(gq + 1, false)) { ok = false; break; }
            }
            if (t + 2 == n_q) tc5::mma_commit(bar(B3_KVE));
          }
        }
        if (!ok) break;
        tc5::mma_commit(bar(B_ACC));
        g0 += n_q;
        ++it;
      }
    }
  } else {
    regs_softmax<88>();
    // ------------------------------------------------------------------ one thread per key row and query half
    const int qd = warp & 3;
    const int wg = (warp - 4) >> 2;    // group g: queries 64 g .. 64 g + 63 of every tile
    const int row = qd * 32 + lane;
    const uint32_t tlane = tmem_base + ((uint32_t)(qd * 32) << 16);
    const float sl = p.scale * kLog2e;
    const uint64_t sl2 = f2_pack(sl, sl);
    const uint32_t prow0 = base + OFF_PT + (uint32_t)wg * PANEL + (uint32_t)row * 128u;
    const uint32_t swz = (uint32_t)(row & 7);
    int g0 = 0, it = 0;
    bool ok = true;
    for (int w = 0; w < n_waves && ok; ++w) {
      const int item = item_at(w);
      if (item >= n_items) continue;
      int kt, bh;
      order.decode(item, kt, bh);
      const int b = bh / p.heads, h = bh - b * p.heads;
      const int k0 = kt * 128;
      const int grow = k0 + row;
      const int t_first = p.causal ? kt : 0;
      const int n_q = nq_all - t_first;
      for (int t = 0; t < n_q; ++t) {
        const int gq = g0 + t;
        const int so = gq % ND;
        const int qrow0 = (t_first + t) * 128 + wg * 64;    // first query of this group's half
        if (!wait_warp(bar(B_OF + so), (uint32_t)(gq / ND) & 1u)) { ok = false; break; }
        if (!wait_warp(bar(B_SF), (uint32_t)gq & 1u)) { ok = false; break; }
        tc5::fence_after_sync();
        const bool need_mask = p.causal && (qrow0 < k0 + 128);
        const float4* nlse = reinterpret_cast<const float4*>(s_lse + so * 128 + wg * 64);
        const float4* ndlt = reinterpret_cast<const float4*>(s_delta + so * 128 + wg * 64);
        uint32_t rs[2][32], rd[2][32];
        tc5::tmem_ld32(tlane + TM_ST + (uint32_t)wg * 64u, rs[0]);
        tc5::tmem_ld32(tlane + TM_ST + (uint32_t)wg * 64u + 32u, rs[1]);
        tc5::tmem_ld_wait();
        if (!PT_TMEM) {
          tc5::fence_before_sync();
          __syncwarp();
          if (lane == 0) tc5::mbar_arrive(bar(B_SE));    // the score tile may take the next tile
        }
        const uint32_t tdp = tlane + TM_DPT + (uint32_t)(gq % NB) * 128u + (uint32_t)wg * 64u;
        const uint32_t prow = prow0 + (uint32_t)(gq % NB) * TILE_P;
        // P^T = exp2(s * sl - lse[query]), dS^T = P^T * (dP^T - delta[query]); two queries per instruction.  s_lse and s_delta
        // hold the negated values, so both enter as plain addends.
#pragma unroll
        for (int i = 0; i < 64; i += 4) {
          const float4 l4 = nlse[i >> 2];
          uint32_t* q = &rs[i >> 5][i & 31];
          const float2 x = f2_unpack(f2_fma(f2_pack(__uint_as_float(q[0]), __uint_as_float(q[1])), sl2, f2_pack(l4.x, l4.y)));
          const float2 z = f2_unpack(f2_fma(f2_pack(__uint_as_float(q[2]), __uint_as_float(q[3])), sl2, f2_pack(l4.z, l4.w)));
          q[0] = __float_as_uint(ex2(x.x));
          q[1] = __float_as_uint(ex2(x.y));
          q[2] = __float_as_uint(ex2(z.x));
          q[3] = __float_as_uint(ex2(z.y));
        }
        if (need_mask) {    // queries before the key
#pragma unroll
          for (int i = 0; i < 64; ++i)
            if (i < grow - qrow0) rs[i >> 5][i & 31] = 0u;
        }
        uint32_t pk[32];
#pragma unroll
        for (int i = 0; i < 64; i += 2) pk[i >> 1] = pack_bf16(__uint_as_float(rs[i >> 5][i & 31]), __uint_as_float(rs[i >> 5][(i & 31) + 1]));
        if (PT_TMEM) {
          tc5::tmem_st32(tlane + TM_ST + (uint32_t)wg * 64u, pk);
          tc5::tmem_st_wait();
          tc5::fence_before_sync();
        } else {
          // dV of the last tile that used this P^T buffer has read it
          if (gq >= NB && !wait_warp(bar(B_PE + gq % NB), (uint32_t)(gq / NB - 1) & 1u)) { ok = false; break; }
#pragma unroll
          for (int g = 0; g < 8; ++g)    // 16-byte chunk g = queries 8g .. 8g+7 of this half
            st_shared_v4(prow + ((((uint32_t)g) ^ swz) << 4), pk[4 * g], pk[4 * g + 1], pk[4 * g + 2], pk[4 * g + 3]);
          fence_async_smem();
        }
        __syncwarp();
        if (lane == 0) tc5::mbar_arrive(bar(B_PP + gq % NB));    // dV may start while dS^T is being computed
        if (!wait_warp(bar(B_DF + gq % NB), (uint32_t)(gq / NB) & 1u)) { ok = false; break; }
        tc5::fence_after_sync();
        tc5::tmem_ld32(tdp, rd[0]);
        tc5::tmem_ld32(tdp + 32u, rd[1]);
        tc5::tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 64; i += 4) {
          const float4 d4 = ndlt[i >> 2];
          const uint32_t *q = &rs[i >> 5][i & 31], *d = &rd[i >> 5][i & 31];
          const float2 a = f2_unpack(f2_mul(f2_pack(__uint_as_float(q[0]), __uint_as_float(q[1])),
                                            f2_add(f2_pack(__uint_as_float(d[0]), __uint_as_float(d[1])), f2_pack(d4.x, d4.y))));
          const float2 c = f2_unpack(f2_mul(f2_pack(__uint_as_float(q[2]), __uint_as_float(q[3])),
                                            f2_add(f2_pack(__uint_as_float(d[2]), __uint_as_float(d[3])), f2_pack(d4.z, d4.w))));
          pk[i >> 1] = pack_bf16(a.x, a.y);
          pk[(i >> 1) + 1] = pack_bf16(c.x, c.y);
        }
        tc5::tmem_st32(tdp, pk);
        tc5::tmem_st_wait();
        tc5::fence_before_sync();
        __syncwarp();
        if (lane == 0) {
          tc5::mbar_arrive(bar(B_PF + gq % NB));
          tc5::mbar_arrive(bar(B_OE + so));
        }
      }
      if (!ok || !wait_warp(bar(B_ACC), (uint32_t)it & 1u)) { ok = false; break; }
      tc5::fence_after_sync();
      // group 0 stores dV, group 1 stores dK: read the whole accumulator first, so that it is free for the next item
      __nv_bfloat16* dst = wg == 0 ? p.dv + (int64_t)b * p.dv_sb + (int64_t)(k0 + qd * 32) * p.dv_ss + (int64_t)h * p.dv_sh
                                   : p.dk + (int64_t)b * p.dk_sb + (int64_t)(k0 + qd * 32) * p.dk_ss + (int64_t)h * p.dk_sh;
      const float f = wg == 0 ? 1.0f : p.scale;
      const uint32_t tsrc = tlane + (wg == 0 ? TM_DV : TM_DK);
      uint32_t acc[D / 32][32];
#pragma unroll
      for (int c = 0; c < D / 32; ++c) tc5::tmem_ld32(tsrc + (uint32_t)c * 32u, acc[c]);
      tc5::tmem_ld_wait();
      tc5::fence_before_sync();
      __syncwarp();
      if (lane == 0) tc5::mbar_arrive(bar(B3_OE));
#pragma unroll
      for (int c = 0; c < D / 32; c += 2) {
        float v[64];
#pragma unroll
        for (int i = 0; i < 64; ++i) v[i] = __uint_as_float(acc[c + (i >> 5)][i & 31]) * f;
        st_rows64(dst + c * 32, wg == 0 ? p.dv_ss : p.dk_ss, p.seqlen - k0 - qd * 32, v);
      }
      g0 += n_q;
      ++it;
    }
  }

  __syncwarp();
  if (*abort_flag) __nanosleep(200000);
  tc5::fence_before_sync();
  __syncthreads();
  tc5::fence_after_sync();
  if (warp == 1) tc5::tmem_dealloc(tmem_base, TM_COLS);
}

// ---- host side -----------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* sym = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess) {
      fn = reinterpret_cast<EncodeTiledFn>(sym);
    }
  });
  return fn;
}

struct Map4Key {
  const void* ptr;
  int64_t sb, ss, sh;
  int batch, heads, seqlen, head_dim, box_rows;
  bool operator==(const Map4Key& o) const {
    return ptr == o.ptr && sb == o.sb && ss == o.ss && sh == o.sh && batch == o.batch && heads == o.heads && seqlen == o.seqlen &&
           head_dim == o.head_dim && box_rows == o.box_rows;
  }
};
struct Map4Hash {
  size_t operator()(const Map4Key& k) const {
    size_t hsh = reinterpret_cast<size_t>(k.ptr);
    auto mix = [&](size_t v) { hsh ^= v * 0x9e3779b97f4a7c15ull + (hsh << 6) + (hsh >> 2); };
    mix((size_t)k.sb); mix((size_t)k.ss); mix((size_t)k.sh); mix((size_t)k.batch); mix((size_t)k.heads); mix((size_t)k.seqlen);
    mix((size_t)k.head_dim); mix((size_t)k.box_rows);
    return hsh;
  }
};

// Tensor map over a bf16 [batch, seq, head, head_dim] view given by element strides; the box is
// [box_rows sequence positions][64 elements] of one head (one 128-byte-swizzled panel).
int make_map4(const void* ptr, int batch, int heads, int seqlen, int head_dim, int64_t sb, int64_t ss, int64_t sh, int box_rows,
              CUtensorMap* out) {
  static std::unordered_map<Map4Key, CUtensorMap, Map4Hash> cache;
  static std::mutex mu;
  Map4Key key{ptr, sb, ss, sh, batch, heads, seqlen, head_dim, box_rows};
  {
    std::lock_guard<std::mutex> lk(mu);
    auto it = cache.find(key);
    if (it != cache.end()) {
      *out = it->second;
      return MSAMP_OK;
    }
  }
  EncodeTiledFn fn = encode_fn();
  if (!fn) {
    msamp_set_error("cuTensorMapEncodeTiled is not available from the driver");
    return MSAMP_ETMAP;
  }
  // The driver call needs a current context.  A thread whose first CUDA call this is (autograd runs backward in threads of its
  // own) has none yet; setting the device that it is on makes the primary one current.
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaSetDevice(dev);
  if (e != cudaSuccess) {
    msamp_set_error("attention: no CUDA context: %s", cudaGetErrorString(e));
    return MSAMP_ELAUNCH;
  }
  // A dimension of extent 1 still needs a valid (16-byte multiple) stride.
  cuuint64_t dims[4] = {(cuuint64_t)head_dim, (cuuint64_t)heads, (cuuint64_t)seqlen, (cuuint64_t)batch};
  cuuint64_t strides[3] = {(cuuint64_t)sh * 2, (cuuint64_t)ss * 2, (cuuint64_t)sb * 2};
  for (int i = 0; i < 3; ++i)
    if (strides[i] == 0) strides[i] = 256;
  cuuint32_t box[4] = {64, 1, (cuuint32_t)box_rows, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(ptr), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    msamp_set_error("cuTensorMapEncodeTiled (attention) failed with %d (ptr=%p b=%d h=%d s=%d strides=%lld,%lld,%lld)", (int)r, ptr,
                    batch, heads, seqlen, (long long)sb, (long long)ss, (long long)sh);
    return MSAMP_ETMAP;
  }
  std::lock_guard<std::mutex> lk(mu);
  if (cache.size() > 4096) cache.clear();
  cache[key] = *out;
  return MSAMP_OK;
}

template <typename K>
int set_smem(K kernel, int bytes) {
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e != cudaSuccess) {
    msamp_set_error("cudaFuncSetAttribute(%d bytes): %s", bytes, cudaGetErrorString(e));
    return MSAMP_ELAUNCH;
  }
  return MSAMP_OK;
}

}    // namespace

// Heads per group of the persistent kernels' work lists: at least four waves of items, and as many as keep two operands of
// all of them within 48 MB of the 126 MB L2 (fewer groups balance better: a group's longest rows start anew).
static int item_group(int seqlen, int head_dim) {
  const int n = (seqlen + 127) / 128;
  const int64_t fit = (48LL << 20) / ((int64_t)seqlen * head_dim * 4);
  const int waves = 4 * msamp_sm_count() / n;
  return (int)(fit > waves ? (fit < (1 << 20) ? fit : (1 << 20)) : (waves > 1 ? waves : 1));
}

// A tensor map has no zero stride: views that repeat a batch, position or head (`expand`) take the mma.sync kernels.
static bool has_repeats(const int64_t* strides, int tensors, int batch, int heads, int seqlen) {
  for (int t = 0; t < tensors; ++t)
    if ((batch > 1 && strides[3 * t] == 0) || (seqlen > 1 && strides[3 * t + 1] == 0) || (heads > 1 && strides[3 * t + 2] == 0)) return true;
  return false;
}

// Short rows: the mma.sync kernels of attention.cu, whose 64-row tiles pad less and whose small CTAs share an SM, where they are the
// faster ones.  tcgen05 time over mma.sync time, causal / full, at heads * batch = 12, 96 and 768:
//   head  rows      forward                          backward
//   64    16        2.0/2.0  2.1/2.1  2.1/2.1        1.8/1.7  1.7/1.7  2.4/2.4
//   64    64        1.9/2.0  1.9/2.2  1.9/2.0        1.4/1.4  1.4/1.3  1.5/1.4
//   64    128       1.8/1.6  1.4/1.4  1.0/0.8        1.1/1.1  0.8/0.8  0.8/0.6
//   64    129       1.4/1.5  1.4/1.4  1.3/1.1        1.2/1.1  1.1/1.2  1.0/0.9
//   64    256       1.3/1.2  1.0/1.0  0.9/0.7        0.9/0.8  0.6/0.8  0.6/0.5
//   64    320       1.1/1.2  0.9/0.9  1.0/0.9        0.9/0.8  0.7/0.6  0.7/0.6
//   64    384       1.1/1.1  0.9/0.8  0.9/0.6        0.8/0.7  0.5/0.4  0.6/0.5
//   128   16        1.1/1.1  1.1/1.2  1.1/1.1        1.3/1.3  1.3/1.3  1.5/1.5
//   128   64        1.1/1.2  1.2/1.2  1.1/1.2        1.1/1.1  1.1/1.0  1.1/1.0
// Above 64 rows the line depends on how many of the persistent kernels' items (128-row tiles) there are for each SM.  Head size 128
// stays on tcgen05 there: its rows are split into two running maxima, which mma.sync does not do (see kSplitRows).
static bool short_rows(int seqlen, int head_dim, int64_t heads, bool backward) {
  if (heads > 65535) return false;    // grid.y of those kernels
  if (seqlen <= 64) return true;
  if (head_dim != 64) return false;
  const int64_t sms = msamp_sm_count(), items = heads * ((seqlen + 127) / 128), waves = (items + sms - 1) / sms;
  const bool idle = waves <= 2 && 10 * items < 7 * waves * sms;    // SMs without an item in the last wave
  if (backward) {
    if (seqlen <= 128) return 2 * items <= sms || (idle && waves == 2 && seqlen <= 96);
    return idle && seqlen <= 192;
  }
  if (seqlen <= 128) return items <= 4 * sms;
  if (seqlen <= 192) return true;    // three 64-row tiles against two of 128
  if (seqlen <= 320) return 2 * items <= 3 * sms;
  return seqlen <= 384 && 2 * items <= sms;
}

extern "C" int msamp_attention_fwd(const void*, const void*, const void*, void*, float*, const int64_t*, int, int, int, int, float, int, void*);
extern "C" int msamp_attention_bwd(const void*, const void*, const void*, const void*, const float*, const void*, void*, void*, void*, float*,
                                   const int64_t*, int, int, int, int, float, int, void*);

// Head size 128, up to this many rows: the kernels that give each half of the 128 keys of a tile a maximum and an accumulator of its
// own, attn_fwd_tm_kernel while the items fit the SMs once (its prologue is shorter: 12 heads of 200, 8.0 -> 7.2 us against
// attn_fwd_split_kernel) and attn_fwd_split_kernel for longer lists.  attn_fwd_ps_kernel is up to 1.5 times as fast there (768 heads of
// 128: 20 against 30 us), but has room for one accumulator only.  Its P is then relative to the maximum of all 128 keys, one
// probability that is exactly 1 instead of two, and with few tiles the output is further from 64 bits: 0.00216 against 0.00210 at
// 128 rows (relative 2-norm, of it 0.0017 from rounding the output), equal from 385 to 450 rows on, closer beyond (0.00220 against
// 0.00227 at 384, not causal).  Up to 64 rows the two are the same.
constexpr int kSplitRows = 448;

// Same contract as msamp_attention_fwd (attention.cu), head_dim 64 or 128: strides are the (batch, seq, head)
// element strides of q, k, v, o; every pointer 16-byte aligned, every stride a multiple of 8 elements.
// All checks and tensor maps come before the first launch, so that a call that is refused has queued nothing.
MSAMP_API int msamp_attention_tc_fwd(const void* q, const void* k, const void* v, void* o, float* lse, const int64_t* strides, int batch,
                                     int heads, int seqlen, int head_dim, float scale, int causal, void* stream_) {
  MSAMP_REQUIRE(head_dim == 64 || head_dim == 128, "attention (tcgen05): head_dim must be 64 or 128 (got %d)", head_dim);
  MSAMP_REQUIRE(batch > 0 && heads > 0 && seqlen > 0, "attention: empty problem");
  MSAMP_REQUIRE(aligned16(q) && aligned16(k) && aligned16(v) && aligned16(o), "attention: q, k, v and o must be 16-byte aligned");
  for (int i = 0; i < 12; ++i) MSAMP_REQUIRE(strides[i] % 8 == 0, "attention: stride %d is not a multiple of 8 elements", i);
  if (has_repeats(strides, 3, batch, heads, seqlen) || short_rows(seqlen, head_dim, (int64_t)batch * heads, false))
    return msamp_attention_fwd(q, k, v, o, lse, strides, batch, heads, seqlen, head_dim, scale, causal, stream_);
  // MSAMP_ATTN_FWD_SMEM=1 selects the kernel with 64-key score tiles and P in shared memory (default: 128-key score
  // tiles, P in tensor memory), MSAMP_ATTN_FWD_PERSIST=0 one CTA per (query tile, batch, head) instead of persistent CTAs.
  static const bool smem_env = [] { const char* e = getenv("MSAMP_ATTN_FWD_SMEM"); return e && e[0] == '1'; }();
  static const bool persist_env = [] { const char* e = getenv("MSAMP_ATTN_FWD_PERSIST"); return !(e && e[0] == '0'); }();
  const int n_qt = (seqlen + 127) / 128;
  const int n_items = n_qt * batch * heads;
  const int ctas = n_items < msamp_sm_count() ? n_items : msamp_sm_count();
  enum { SMEM, TM, SPLIT, PS } kind = PS;
  if (head_dim == 128) {
    if (smem_env) kind = SMEM;
    else if (!persist_env || (seqlen <= kSplitRows && n_items <= ctas)) kind = TM;
    else if (seqlen > 64 && seqlen <= kSplitRows) kind = SPLIT;
  }
  const int k_rows = kind == SMEM ? 64 : 128, v_rows = kind == PS ? 128 : 64;
  CUtensorMap mq, mk, mv;
  int rc;
  if ((rc = make_map4(q, batch, heads, seqlen, head_dim, strides[0], strides[1], strides[2], 128, &mq))) return rc;
  if ((rc = make_map4(k, batch, heads, seqlen, head_dim, strides[3], strides[4], strides[5], k_rows, &mk))) return rc;
  if ((rc = make_map4(v, batch, heads, seqlen, head_dim, strides[6], strides[7], strides[8], v_rows, &mv))) return rc;
  TcParams p = {};
  p.o = (__nv_bfloat16*)o; p.lse = lse;
  p.o_sb = strides[9]; p.o_ss = strides[10]; p.o_sh = strides[11];
  p.batch = batch; p.heads = heads; p.seqlen = seqlen; p.causal = causal; p.scale = scale;
  p.status = msamp_device_status_ptr();
  p.group = item_group(seqlen, head_dim);
  cudaStream_t stream = (cudaStream_t)stream_;
  dim3 grid(n_qt, batch * heads);
  if (kind == SMEM) {
    if ((rc = set_smem(attn_fwd_tc_kernel, fwd::SMEM))) return rc;
    attn_fwd_tc_kernel<<<grid, kTcThreads, fwd::SMEM, stream>>>(mq, mk, mv, p);
    return msamp_check_launch("attn_fwd_tc_kernel");
  }
  if (kind == TM) {
    if ((rc = set_smem(attn_fwd_tm_kernel, fwd2::SMEM))) return rc;
    attn_fwd_tm_kernel<<<grid, kTcThreads, fwd2::SMEM, stream>>>(mq, mk, mv, p);
    return msamp_check_launch("attn_fwd_tm_kernel");
  }
  if (kind == SPLIT) {
    if ((rc = set_smem(attn_fwd_split_kernel, fwd2s::SMEM3))) return rc;
    attn_fwd_split_kernel<<<ctas, kTcThreads, fwd2s::SMEM3, stream>>>(mq, mk, mv, p, n_qt, n_items);
    return msamp_check_launch("attn_fwd_split_kernel");
  }
  if (head_dim == 128) {
    if ((rc = set_smem(attn_fwd_ps_kernel<128>, fwd3::Cfg<128>::SMEM))) return rc;
    attn_fwd_ps_kernel<128><<<ctas, kPsThreads, fwd3::Cfg<128>::SMEM, stream>>>(mq, mk, mv, p, n_qt, n_items);
  } else {
    if ((rc = set_smem(attn_fwd_ps_kernel<64>, fwd3::Cfg<64>::SMEM))) return rc;
    attn_fwd_ps_kernel<64><<<ctas, kPsThreads, fwd3::Cfg<64>::SMEM, stream>>>(mq, mk, mv, p, n_qt, n_items);
  }
  return msamp_check_launch("attn_fwd_ps_kernel");
}

// Same contract as msamp_attention_bwd (attention.cu), head_dim 64 or 128.
MSAMP_API int msamp_attention_tc_bwd(const void* q, const void* k, const void* v, const void* o, const float* lse, const void* d_o,
                                     void* dq, void* dk, void* dv, float* delta, const int64_t* strides, int batch, int heads,
                                     int seqlen, int head_dim, float scale, int causal, void* stream_) {
  MSAMP_REQUIRE(head_dim == 64 || head_dim == 128, "attention (tcgen05): head_dim must be 64 or 128 (got %d)", head_dim);
  MSAMP_REQUIRE(batch > 0 && heads > 0 && seqlen > 0, "attention: empty problem");
  MSAMP_REQUIRE(aligned16(q) && aligned16(k) && aligned16(v) && aligned16(o) && aligned16(d_o) && aligned16(dq) && aligned16(dk) && aligned16(dv),
                "attention: q, k, v, o, dO and the gradients must be 16-byte aligned");
  for (int i = 0; i < 24; ++i) MSAMP_REQUIRE(strides[i] % 8 == 0, "attention: stride %d is not a multiple of 8 elements", i);
  if (has_repeats(strides, 5, batch, heads, seqlen) || short_rows(seqlen, head_dim, (int64_t)batch * heads, true))
    return msamp_attention_bwd(q, k, v, o, lse, d_o, dq, dk, dv, delta, strides, batch, heads, seqlen, head_dim, scale, causal, stream_);
  // MSAMP_ATTN_BWD_SMEM=1 selects the kernels with 64-wide score tiles and the second operand in shared memory,
  // MSAMP_ATTN_BWD_PERSIST=0 one CTA per (tile, batch, head) instead of persistent CTAs over the work items
  static const bool smem_env = [] { const char* e = getenv("MSAMP_ATTN_BWD_SMEM"); return e && e[0] == '1'; }();
  static const bool persist_env = [] { const char* e = getenv("MSAMP_ATTN_BWD_PERSIST"); return !(e && e[0] == '0'); }();
  const bool smem_operands = smem_env && head_dim == 128, persistent = persist_env || head_dim == 64;
  // boxes of 128 rows throughout, except for the operand that the 64-wide kernels stream
  CUtensorMap mq, mk, mv, mdo, mq64, mk64, mv64, mdo64;
  int rc;
  if ((rc = make_map4(q, batch, heads, seqlen, head_dim, strides[0], strides[1], strides[2], 128, &mq))) return rc;
  if ((rc = make_map4(k, batch, heads, seqlen, head_dim, strides[3], strides[4], strides[5], 128, &mk))) return rc;
  if ((rc = make_map4(v, batch, heads, seqlen, head_dim, strides[6], strides[7], strides[8], 128, &mv))) return rc;
  if ((rc = make_map4(d_o, batch, heads, seqlen, head_dim, strides[12], strides[13], strides[14], 128, &mdo))) return rc;
  if (smem_operands) {
    if ((rc = make_map4(q, batch, heads, seqlen, head_dim, strides[0], strides[1], strides[2], 64, &mq64))) return rc;
    if ((rc = make_map4(k, batch, heads, seqlen, head_dim, strides[3], strides[4], strides[5], 64, &mk64))) return rc;
    if ((rc = make_map4(v, batch, heads, seqlen, head_dim, strides[6], strides[7], strides[8], 64, &mv64))) return rc;
    if ((rc = make_map4(d_o, batch, heads, seqlen, head_dim, strides[12], strides[13], strides[14], 64, &mdo64))) return rc;
  }
  cudaStream_t stream = (cudaStream_t)stream_;
  {
    DeltaParams d = {};
    d.o = (const __nv_bfloat16*)o; d.d_o = (const __nv_bfloat16*)d_o; d.delta = delta;
    d.o_sb = strides[9]; d.o_ss = strides[10]; d.o_sh = strides[11];
    d.do_sb = strides[12]; d.do_ss = strides[13]; d.do_sh = strides[14];
    d.batch = batch; d.heads = heads; d.seqlen = seqlen;
    const int64_t rows = (int64_t)batch * heads * seqlen;
    const int per_cta = 2 * 256 / (head_dim / 8);
    const unsigned blocks = (unsigned)((rows + per_cta - 1) / per_cta);
    if (head_dim == 128) attn_delta_tc_kernel<128><<<blocks, 256, 0, stream>>>(d);
    else                 attn_delta_tc_kernel<64><<<blocks, 256, 0, stream>>>(d);
  }
  TcParams p = {};
  p.lse = const_cast<float*>(lse); p.delta = delta;
  p.dq = (__nv_bfloat16*)dq; p.dk = (__nv_bfloat16*)dk; p.dv = (__nv_bfloat16*)dv;
  p.dq_sb = strides[15]; p.dq_ss = strides[16]; p.dq_sh = strides[17];
  p.dk_sb = strides[18]; p.dk_ss = strides[19]; p.dk_sh = strides[20];
  p.dv_sb = strides[21]; p.dv_ss = strides[22]; p.dv_sh = strides[23];
  p.batch = batch; p.heads = heads; p.seqlen = seqlen; p.causal = causal; p.scale = scale;
  p.status = msamp_device_status_ptr();
  p.group = item_group(seqlen, head_dim);
  const int n_t = (seqlen + 127) / 128;    // key tiles of dK / dV, query tiles of dQ
  const int n_items = n_t * batch * heads;
  const int ctas = n_items < msamp_sm_count() ? n_items : msamp_sm_count();
  dim3 grid(n_t, batch * heads);
  if (smem_operands) {
    if ((rc = set_smem(attn_bwd_dkdv_tc_kernel, dkv::SMEM))) return rc;
    attn_bwd_dkdv_tc_kernel<<<grid, kTcThreads, dkv::SMEM, stream>>>(mq64, mk, mv, mdo64, p);
    if ((rc = set_smem(attn_bwd_dq_tc_kernel, dqk::SMEM))) return rc;
    attn_bwd_dq_tc_kernel<<<grid, kTcThreads, dqk::SMEM, stream>>>(mq, mk64, mv64, mdo, p);
  } else if (!persistent) {
    if ((rc = set_smem(attn_bwd_dkdv_tm_kernel, dkv2::SMEM))) return rc;
    attn_bwd_dkdv_tm_kernel<<<grid, kTcThreads, dkv2::SMEM, stream>>>(mq, mk, mv, mdo, p);
    if ((rc = set_smem(attn_bwd_dq_tm_kernel, dqk2::SMEM))) return rc;
    attn_bwd_dq_tm_kernel<<<grid, kTcThreads, dqk2::SMEM, stream>>>(mq, mk, mv, mdo, p);
  } else if (head_dim == 128) {
    if ((rc = set_smem(attn_bwd_dkdv_ps_kernel<128>, dkv3::Cfg<128>::SMEM))) return rc;
    attn_bwd_dkdv_ps_kernel<128><<<ctas, kPsThreads, dkv3::Cfg<128>::SMEM, stream>>>(mq, mk, mv, mdo, p, n_t, n_items);
    if ((rc = set_smem(attn_bwd_dq_ps_kernel<128>, dqk3::Cfg<128>::SMEM))) return rc;
    attn_bwd_dq_ps_kernel<128><<<ctas, kPsThreads, dqk3::Cfg<128>::SMEM, stream>>>(mq, mk, mv, mdo, p, n_t, n_items);
  } else {
    if ((rc = set_smem(attn_bwd_dkdv_ps_kernel<64>, dkv3::Cfg<64>::SMEM))) return rc;
    attn_bwd_dkdv_ps_kernel<64><<<ctas, kPsThreads, dkv3::Cfg<64>::SMEM, stream>>>(mq, mk, mv, mdo, p, n_t, n_items);
    if ((rc = set_smem(attn_bwd_dq_ps_kernel<64>, dqk3::Cfg<64>::SMEM))) return rc;
    attn_bwd_dq_ps_kernel<64><<<ctas, kPsThreads, dqk3::Cfg<64>::SMEM, stream>>>(mq, mk, mv, mdo, p, n_t, n_items);
  }
  return msamp_check_launch("attn_bwd_tc kernels");
}
