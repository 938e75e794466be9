// Flash attention forward on the 5th-generation tensor cores (tcgen05 + TMEM), fed by TMA: a kernel with two query tiles
// per CTA (head sizes 64 and 128) and one with a single tile whose key blocks alternate between two groups of warps (256).
//
// Scores are computed by tcgen05.mma into tensor memory; a thread takes one query row (tcgen05.ld hands it its row, so
// maximum and sum need no exchange), reads its scores once into registers, and writes P (bf16) back to tensor memory, where
// it is the A operand of the second product.  O stays in tensor memory for the whole sweep and is rescaled only when
// the running max has moved by more than 2^8 (P stays within bf16/fp32 range; the final division by the row sum makes
// the result independent of the reference point).  Blocks that no mask touches take a path without position arithmetic.
// V is consumed MN-major straight from its row-major [kv, head_dim] tile: no transposes anywhere.
//
// Semantics (compiler/mesh_compiler/operations.py:7081-7166): blockwise online softmax with (m, s, acc)
// merging, causal and sliding-window masks on *logical* positions (q_pos = q_off + i*q_stride,
// k_pos = k_off + j*k_stride, which covers striped context-parallel layouts, :7044-7069), GQA by mapping
// query head h to KV head h / group (:7072-7078); the log-sum-exp is returned so partial results over
// KV chunks (ring attention) can be merged.  Fully masked KV blocks are skipped.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math_constants.h>
#include <cstring>
#include "ops_api.h"
#include "../device/philox.cuh"
#include "../device/ptx.cuh"
#include "../runtime/host_common.h"

namespace mesh {
namespace fa {

constexpr int SM_THREADS = 256;       // 8 softmax warps

struct Params {
  CUtensorMap tmQ, tmK, tmV;          // [sample][row][column], boxes of 64 columns and 128 rows
  CUtensorMap tmK2, tmV2;             // [row][column] over all samples: key blocks that end inside their sample
  __nv_bfloat16* out; long long ldo;  // [B*Tq, H*hd]
  float* lse;                         // [B, H, Tq]
  int B, H, Hkv, Tq, Tk;
  int q_col0, k_col0, v_col0;         // first column of head 0 inside the stored matrices
  int causal, window;
  int q_off, q_stride, k_off, k_stride;
  float scale_log2;                   // softmax scale * log2(e)
  Status* status;
  DropoutKey drop;
  int head_off, heads_total;                    // drop.p == 0: no dropout
};

__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// two fp32 at a time
struct F2 { unsigned long long v; };
__device__ __forceinline__ F2 f2(float lo, float hi) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack(F2 a, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(a.v)); }
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
__device__ __forceinline__ F2 add2(F2 a, F2 b) {
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}

// ------------------------------------------------------------------------------------------------ two query tiles
// Head sizes 64 and 128.  One CTA owns 256 query rows of a head as two tiles of 128; while the softmax warps of one
// tile turn its scores into probabilities, the tensor core runs the products of the other, so neither waits for the
// other's chain.  Tensor memory: S of tile 0 and 1 in columns 0 and 128 (P, as bf16 pairs, overwrites the first half of
// its own S and feeds the second product from there), O of the two tiles from column 256.
//
// Warps 0-3 / 4-7: softmax of tile 0 / 1, one thread per query row (no exchange between threads); warp 8 streams K
// and V through two stages each; warp 9 issues, per key block and tile, O += P V and then S of the next key block: the
// tensor core runs one thread's products in order, so S may overwrite the P that the product before it reads.
// P is never staged in shared memory, which leaves its bandwidth to the operands (a 128 x 128 x 128 product with both
// operands in shared memory reads 64 KB in the 512 cycles it computes: exactly the limit).
//
// Bound by the exponentials: a 128 x 128 block takes 1024 cycles of the special-function units beside 1024 (head size
// 128) or 512 (64) of the tensor pipe.  Measured at one sequence of 8192, 16 heads of 128, causal: 1014 us with one
// tile per CTA and P in shared memory, 250 us with this one (1100 TFLOP/s); heads of 64: 201 us.
constexpr int TT = 128;                               // rows of a tile
constexpr int THREADS2 = 320;

template <int HD>
struct Cfg2 {
  static constexpr int KC = HD / 64;
  static constexpr int TILE = TT * HD * 2;            // Q tile, K block, V block
  static constexpr int SMEM = 6 * TILE + 1024 + 256;
  static constexpr int O_COL0 = 256;
};

// floor(a / b) for b > 0
__device__ __forceinline__ int floor_div(int a, int b) {
  const int q = a / b;
  return q - ((a % b) < 0 ? 1 : 0);
}

template <int HD, bool DROP>
__global__ void __launch_bounds__(THREADS2, 1) flash_fwd2_kernel(const __grid_constant__ Params p) {
  using C = Cfg2<HD>;
  constexpr int KC = C::KC;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t sQ = base, sK = sQ + 2 * C::TILE, sV = sK + 2 * C::TILE, bars = sV + 2 * C::TILE;
  auto bar = [&](int i) { return bars + 8u * i; };
  constexpr int Q_FULL = 0, K_FULL = 1, V_FULL = 3, K_EMPTY = 5, V_EMPTY = 7, S_FULL = 9, P_FULL = 11, O_DONE = 13, P_HALF = 15, N_BARS = 17;
  uint8_t* gen = smem_raw + (base - smem_u32(smem_raw));
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(gen + 6 * C::TILE + 8 * N_BARS);
  volatile int* abort_smem = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // the query blocks with the most visible keys start first (causal: the last ones), so the tail of the grid is short
  const int qb = gridDim.y - 1 - blockIdx.y;
  const int h = blockIdx.x % p.H, b = blockIdx.x / p.H;
  const int hk = h / (p.H / p.Hkv);
  const int q0 = qb * 2 * TT;

  // key blocks visible to each tile (logical positions): [lo[t], hi[t])
  int lo[2], hi[2];
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    const int r0 = q0 + t * TT;
    lo[t] = 0;
    hi[t] = r0 < p.Tq ? (p.Tk + TT - 1) / TT : 0;
    const int pos_lo = p.q_off + r0 * p.q_stride;
    const int pos_hi = p.q_off + (min(r0 + TT, p.Tq) - 1) * p.q_stride;
    if (p.causal) {
      const int kmax = floor_div(pos_hi - p.k_off, p.k_stride);
      hi[t] = kmax < 0 ? 0 : min(hi[t], kmax / TT + 1);
    }
    if (p.window > 0) {
      const int kmin = floor_div(pos_lo - p.window - p.k_off, p.k_stride) + 1;
      lo[t] = max(0, kmin) / TT;
    }
    if (lo[t] >= hi[t]) lo[t] = hi[t] = 0;
  }
  const bool any0 = hi[0] > lo[0], any1 = hi[1] > lo[1];
  const int j_lo = any0 && any1 ? min(lo[0], lo[1]) : any0 ? lo[0] : lo[1];
  const int j_hi = max(hi[0], hi[1]);

  if (threadIdx.x == 0) {
    mbar_init(bar(Q_FULL), 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(bar(K_FULL + s), 1);
      mbar_init(bar(V_FULL + s), 1);
      mbar_init(bar(K_EMPTY + s), 1);
      mbar_init(bar(V_EMPTY + s), 1);
      mbar_init(bar(S_FULL + s), 1);
      mbar_init(bar(P_HALF + s), TT);
      mbar_init(bar(P_FULL + s), TT);
      mbar_init(bar(O_DONE + s), 1);
    }
    *abort_smem = 0;
    fence_mbar_init();
  }
  if (warp == 9) {
    tmem_alloc<1>(smem_u32(tmem_slot), 512);
    tmem_relinquish<1>();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(tmem_slot);

  if (warp == 8) {
    if (lane == 0 && j_hi > j_lo) {
      // ------------------------------------------------------------------ copies
      const int tiles = any1 ? 2 : 1;                  // the second tile may lie past the last query
      mbar_expect_tx(bar(Q_FULL), tiles * C::TILE);
      for (int t = 0; t < tiles; ++t)
        for (int kc = 0; kc < KC; ++kc)
          tma_load_3d(sQ + t * C::TILE + kc * (TT * 128), &p.tmQ, bar(Q_FULL), p.q_col0 + h * HD + kc * 64, q0 + t * TT, b);
      bool ok = true;
      for (int j = j_lo, n = 0; ok && j < j_hi; ++j, ++n) {
        const int s = n & 1;
        // a copy with three coordinates takes longer: 2.5 % of the kernel with heads of 64 when every block used it
        const bool whole = (j + 1) * TT <= p.Tk;
        const int k_row = b * p.Tk + j * TT;
        if (n >= 2) ok = mbar_wait(bar(K_EMPTY + s), ((n >> 1) - 1) & 1, abort_smem, p.status, SITE_SMEM_EMPTY);
        if (!ok) break;
        mbar_expect_tx(bar(K_FULL + s), C::TILE);
        for (int kc = 0; kc < KC; ++kc)
          if (whole) tma_load_2d(sK + s * C::TILE + kc * (TT * 128), &p.tmK2, bar(K_FULL + s), p.k_col0 + hk * HD + kc * 64, k_row);
          else tma_load_3d(sK + s * C::TILE + kc * (TT * 128), &p.tmK, bar(K_FULL + s), p.k_col0 + hk * HD + kc * 64, j * TT, b);
        if (n >= 2) ok = mbar_wait(bar(V_EMPTY + s), ((n >> 1) - 1) & 1, abort_smem, p.status, SITE_SMEM_EMPTY);
        if (!ok) break;
        mbar_expect_tx(bar(V_FULL + s), C::TILE);
        for (int kc = 0; kc < KC; ++kc)
          if (whole) tma_load_2d(sV + s * C::TILE + kc * (TT * 128), &p.tmV2, bar(V_FULL + s), p.v_col0 + hk * HD + kc * 64, k_row);
          else tma_load_3d(sV + s * C::TILE + kc * (TT * 128), &p.tmV, bar(V_FULL + s), p.v_col0 + hk * HD + kc * 64, j * TT, b);
      }
    }
  } else if (warp == 9) {
    if (j_hi > j_lo) {
      // ------------------------------------------------------------------ products: the whole warp runs the loop and one
      // elected lane issues, so that descriptors and addresses stay in uniform registers
      constexpr uint32_t idesc_s = umma_idesc_bf16(TT, TT, 0, 0);
      constexpr uint32_t idesc_o = umma_idesc_bf16(TT, HD, 0, 1);            // B = V is MN-major
      const bool leader = elect_one();
      const uint64_t dq0 = umma_smem_desc(sQ, 16, 1024), dk0 = umma_smem_desc(sK, 16, 1024);
      const uint64_t dv0 = umma_smem_desc(sV, TT * 128, 1024);               // groups of 64 head dims
      auto issue_s = [&](int t, int s) {
        const uint64_t da = dq0 + (uint32_t)(t * (C::TILE >> 4)), db = dk0 + (uint32_t)(s * (C::TILE >> 4));
        if (leader) {
#pragma unroll
          for (int kc = 0; kc < KC; ++kc)
#pragma unroll
            for (int k = 0; k < 4; ++k)
              umma_f16<1>(tmem + t * 128, da + (kc * (TT * 128) + k * 32) / 16, db + (kc * (TT * 128) + k * 32) / 16, idesc_s, (kc | k) ? 1u : 0u);
          umma_commit(bar(S_FULL + t));
        }
      };
      bool ok = mbar_wait_warp(bar(Q_FULL), 0, abort_smem, p.status, SITE_SMEM_FULL);
      if (ok) ok = mbar_wait_warp(bar(K_FULL), 0, abort_smem, p.status, SITE_SMEM_FULL);
      if (ok) {
        tc_fence_after();
        for (int t = 0; t < 2; ++t)
          if (j_lo >= lo[t] && j_lo < hi[t]) issue_s(t, 0);
        if (leader) umma_commit(bar(K_EMPTY));
      }
      int done[2] = {0, 0};                            // key blocks of each tile whose P V has been issued
      for (int j = j_lo, n = 0; ok && j < j_hi; ++j, ++n) {
        const int s = n & 1, sn = s ^ 1;
        ok = mbar_wait_warp(bar(V_FULL + s), (n >> 1) & 1, abort_smem, p.status, SITE_SMEM_FULL);
        const bool more = j + 1 < j_hi;
        if (ok && more) ok = mbar_wait_warp(bar(K_FULL + sn), ((n + 1) >> 1) & 1, abort_smem, p.status, SITE_SMEM_FULL);
        if (!ok) break;
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          if (j >= lo[t] && j < hi[t]) {
            // the first half of the keys while the threads work on the second
            ok = mbar_wait_warp(bar(P_HALF + t), done[t] & 1, abort_smem, p.status, SITE_TMEM_FULL);
            if (!ok) break;
            tc_fence_after();
            const uint64_t db = dv0 + (uint32_t)(s * (C::TILE >> 4));
            const uint32_t first = done[t] ? 1u : 0u;
            if (leader) {
#pragma unroll
              for (int k = 0; k < TT / 32; ++k)
                umma_f16_ts(tmem + C::O_COL0 + t * 128, tmem + t * 128 + k * 8, db + k * 128, idesc_o, k ? 1u : first);
            }
            __syncwarp();
            ok = mbar_wait_warp(bar(P_FULL + t), done[t] & 1, abort_smem, p.status, SITE_TMEM_FULL);
            if (!ok) break;
            tc_fence_after();
            if (leader) {
#pragma unroll
              for (int k = TT / 32; k < TT / 16; ++k)
                umma_f16_ts(tmem + C::O_COL0 + t * 128, tmem + t * 128 + k * 8, db + k * 128, idesc_o, 1u);
              umma_commit(bar(O_DONE + t));
            }
            ++done[t];
          }
          if (t == 1 && leader) umma_commit(bar(V_EMPTY + s));
          if (more && j + 1 >= lo[t] && j + 1 < hi[t]) issue_s(t, sn);
        }
        if (ok && more && leader) umma_commit(bar(K_EMPTY + sn));
        __syncwarp();
      }
    }
  } else {
    // -------------------------------------------------------------------- softmax warps: thread = query row
    const int t = warp >> 2;
    const int row = threadIdx.x & 127;                 // == TMEM lane
    const int qi = q0 + t * TT + row;
    const int qpos = p.q_off + qi * p.q_stride;
    const uint32_t s_addr = tmem + ((uint32_t)((warp & 3) * 32) << 16) + t * 128;
    const uint32_t o_addr = s_addr + C::O_COL0;
    const int n_blocks = hi[t] - lo[t], j0 = lo[t];
    // keys this row sees: indices [k_first, k_end)
    int k_first = 0, k_end = p.Tk;
    if (p.causal) k_end = min(k_end, floor_div(qpos - p.k_off, p.k_stride) + 1);
    if (p.window > 0) k_first = max(0, floor_div(qpos - p.window - p.k_off, p.k_stride) + 1);
    // a block that every row of the tile sees whole needs no mask
    const int r_lo = q0 + t * TT, r_hi = r_lo + TT - 1;
    int full_lo = 0, full_hi = p.Tk;
    if (p.causal) full_hi = min(full_hi, floor_div(p.q_off + r_lo * p.q_stride - p.k_off, p.k_stride) + 1);
    if (p.window > 0) full_lo = max(0, floor_div(p.q_off + r_hi * p.q_stride - p.window - p.k_off, p.k_stride) + 1);
    const float thr = 8.f / p.scale_log2;              // the reference point moves when the max grew by > 2^8
    float m_ref = -CUDART_INF_F, l = 0.f;
    DropoutRow dr;
    bool ok = true;
    for (int it = 0; it < n_blocks; ++it) {
      ok = mbar_wait(bar(S_FULL + t), it & 1, abort_smem, p.status, SITE_TMEM_FULL);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      uint32_t r[4][32];
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld_32x32(s_addr + c * 32, r[c]);
      tmem_ld_wait();
      const int kbase = (j0 + it) * TT;
      if (kbase < full_lo || kbase + TT > full_hi) {
        const int first = k_first - kbase, end = k_end - kbase;
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (c * 32 + i < first || c * 32 + i >= end) r[c][i] = 0xff800000u;     // -inf: exp2 gives an exact zero
      }
      float mxs[4] = {-CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F};
#pragma unroll
      for (int i = 0; i < 32; ++i)
#pragma unroll
        for (int c = 0; c < 4; ++c) mxs[c] = fmaxf(mxs[c], __uint_as_float(r[c][i]));
      const float mx = fmaxf(fmaxf(mxs[0], mxs[1]), fmaxf(mxs[2], mxs[3]));
      float alpha = 1.f;
      if (mx > m_ref + thr) {                          // also the first block with a visible key (m_ref = -inf)
        alpha = ex2_approx((m_ref - mx) * p.scale_log2);          // ex2(-inf) = 0
        m_ref = mx;
      }
      // tcgen05.ld / .st are warp-collective: the decision must be the same for all 32 rows of a warp.  Never for the
      // first block: its product overwrites O.
      if (it > 0 && __any_sync(0xffffffffu, alpha != 1.f)) {
        ok = mbar_wait(bar(O_DONE + t), (it - 1) & 1, abort_smem, p.status, SITE_TMEM_EMPTY);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
#pragma unroll 1
        for (int c = 0; c < HD / 16; ++c) {
          uint32_t o[16];
          tmem_ld_32x16(o_addr + c * 16, o);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
          tmem_st_32x16(o_addr + c * 16, o);
        }
      }
      const float neg_ms = (m_ref == -CUDART_INF_F) ? 0.f : -m_ref * p.scale_log2;
      if (DROP) dr.begin((uint32_t)(b * p.heads_total + p.head_off + h), (uint32_t)qpos);
      const F2 scale2 = f2(p.scale_log2, p.scale_log2), off2 = f2(neg_ms, neg_ms);
      F2 sum2[2] = {f2(0.f, 0.f), f2(0.f, 0.f)};
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t w[16];
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          float x0, x1;
          unpack(fma2(f2(__uint_as_float(r[c][i]), __uint_as_float(r[c][i + 1])), scale2, off2), x0, x1);
          float p0 = ex2_approx(x0), p1 = ex2_approx(x1);
          sum2[(i / 2) & 1] = add2(sum2[(i / 2) & 1], f2(p0, p1));      // the row sum is that of the undropped probabilities
          if (DROP) {
            const uint32_t kpos = (uint32_t)(p.k_off + (kbase + c * 32 + i) * p.k_stride);
            p0 = dr.keep(p.drop, kpos) ? p0 * p.drop.inv_keep : 0.f;
            p1 = dr.keep(p.drop, kpos + (uint32_t)p.k_stride) ? p1 * p.drop.inv_keep : 0.f;
          }
          __nv_bfloat162 hb = __floats2bfloat162_rn(p0, p1);
          w[i / 2] = *reinterpret_cast<uint32_t*>(&hb);
        }
        tmem_st_32x16(s_addr + c * 16, w);             // every score of the row is in registers by now
        if (c == 1 || c == 3) {
          tmem_st_wait();
          tc_fence_before();
          mbar_arrive(bar((c == 1 ? P_HALF : P_FULL) + t));
        }
      }
      float s0, s1;
      unpack(add2(sum2[0], sum2[1]), s0, s1);
      l = l * alpha + s0 + s1;
    }
    // ---- epilogue: O / l -> bf16 rows, log-sum-exp
    if (ok && n_blocks > 0) {
      ok = mbar_wait(bar(O_DONE + t), (n_blocks - 1) & 1, abort_smem, p.status, SITE_TMEM_FULL);
      tc_fence_after();
    }
    ok = __all_sync(0xffffffffu, ok);                  // the TMEM loads below are warp-collective: every lane takes part,
    if (ok) {                                          // only the global stores are predicated on the row being real
      const float inv = l > 0.f ? 1.f / l : 0.f;
      __nv_bfloat16* dst = p.out + ((long long)b * p.Tq + qi) * p.ldo + h * HD;
#pragma unroll 1
      for (int c = 0; c < HD / 32; ++c) {
        uint32_t o[32];
        if (n_blocks > 0) {
          tmem_ld_32x32(o_addr + c * 32, o);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) o[i] = 0;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          uint4 q4;
          __nv_bfloat162* hb = reinterpret_cast<__nv_bfloat162*>(&q4);
#pragma unroll
          for (int i = 0; i < 4; ++i)
            hb[i] = __floats2bfloat162_rn(__uint_as_float(o[8 * j + 2 * i]) * inv, __uint_as_float(o[8 * j + 2 * i + 1]) * inv);
          if (qi < p.Tq) *reinterpret_cast<uint4*>(dst + c * 32 + j * 8) = q4;
        }
      }
      if (p.lse && qi < p.Tq)
        p.lse[((long long)b * p.H + h) * p.Tq + qi] =
            l > 0.f ? (m_ref * p.scale_log2 + log2f(l)) * 0.6931471805599453f : -CUDART_INF_F;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 9) {
    tc_fence_after();
    tmem_dealloc<1>(tmem, 512);
  }
}

// ------------------------------------------------------------------------------------------------ heads of 256
// The output of one tile takes half of the tensor memory, so there is room for one query tile.  Its key blocks go to the two
// groups of softmax warps in turn: blocks 0, 2, .. have their scores in columns 0.. and belong to warps 0-3 (a thread per
// query row), blocks 1, 3, .. in columns 128.. to warps 4-7, so the exponentials of one block run under those of the next
// and under the products of both.  What the groups share is the reference point of a row: a group compares its block's
// maximum with the point that the other one left in shared memory for the block before (an mbarrier per direction), and a
// thread brings its own row sum to the current point when it comes around.  K and V arrive as halves of 128 x 128 in a ring
// of five 32 KB slots, in the order the products use them: K0 K1 V0 K2 V1 ...
//
// Bound by the 64 bytes a cycle that an SM takes in: 128 KB of K and V per block of keys, 2048 cycles of products.
// Measured at eight sequences of 1024, 8 query heads over 2 KV heads, causal with a window of 512: 115 us with one group of
// blocks in turn and P in shared memory, 57.8 us with this one.
struct Cfg256 {
  static constexpr int HD = 256;
  static constexpr int Q_BYTES = TT * HD * 2, SLOT = TT * 128 * 2, SLOTS = 5;
  static constexpr int N_BARS = 1 + 2 * SLOTS + 10;
  static constexpr int XCHG = 4 * TT * 4;             // reference points of two blocks, row sums of two groups
  static constexpr int SMEM = Q_BYTES + SLOTS * SLOT + XCHG + 8 * N_BARS + 16;     // no room to align by hand
  static constexpr int O_COL0 = 256;
};

template <bool DROP>
__global__ void __launch_bounds__(THREADS2, 1) flash_fwd256_kernel(const __grid_constant__ Params p) {
  using C = Cfg256;
  constexpr int HD = C::HD;
  extern __shared__ __align__(1024) uint8_t smem_al[];
  const uint32_t base = smem_u32(smem_al);
  if (base & 1023u) {                                  // the swizzled tiles need it; nothing is placed before them
    if (threadIdx.x == 0) status_record(p.status, MESH_ALIGN, SITE_NONE, 1024, base);
    return;
  }
  const uint32_t sQ = base, ring = sQ + C::Q_BYTES;
  float* m_s = reinterpret_cast<float*>(smem_al + C::Q_BYTES + C::SLOTS * C::SLOT);        // [block & 1][row]
  float* l_s = m_s + 2 * TT;                                                               // [group][row]
  const uint32_t bars = ring + C::SLOTS * C::SLOT + C::XCHG;
  auto bar = [&](int i) { return bars + 8u * i; };
  constexpr int Q_FULL = 0, FULL = 1, EMPTY = FULL + C::SLOTS, S_FULL = EMPTY + C::SLOTS, P_HALF = S_FULL + 2, P_FULL = P_HALF + 2,
                M_READY = P_FULL + 2, O_DONE = M_READY + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem_al + (bars - base) + 8 * C::N_BARS);
  volatile int* abort_smem = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int qb = gridDim.y - 1 - blockIdx.y;           // the query blocks with the most visible keys start first
  const int h = blockIdx.x % p.H, b = blockIdx.x / p.H;
  const int hk = h / (p.H / p.Hkv);
  const int q0 = qb * TT;
  // key blocks visible to the tile (logical positions): n_blocks from j0
  int j0 = 0, j_hi = (p.Tk + TT - 1) / TT;
  {
    const int pos_lo = p.q_off + q0 * p.q_stride;
    const int pos_hi = p.q_off + (min(q0 + TT, p.Tq) - 1) * p.q_stride;
    if (p.causal) {
      const int kmax = floor_div(pos_hi - p.k_off, p.k_stride);
      j_hi = kmax < 0 ? 0 : min(j_hi, kmax / TT + 1);
    }
    if (p.window > 0) j0 = max(0, floor_div(pos_lo - p.window - p.k_off, p.k_stride) + 1) / TT;
  }
  const int n_blocks = max(0, j_hi - j0);

  if (threadIdx.x == 0) {
    mbar_init(bar(Q_FULL), 1);
    for (int s = 0; s < C::SLOTS; ++s) {
      mbar_init(bar(FULL + s), 1);
      mbar_init(bar(EMPTY + s), 1);
    }
    for (int g = 0; g < 2; ++g) {
      mbar_init(bar(S_FULL + g), 1);
      mbar_init(bar(P_HALF + g), TT);
      mbar_init(bar(P_FULL + g), TT);
      mbar_init(bar(M_READY + g), TT);
      mbar_init(bar(O_DONE + g), 1);
    }
    *abort_smem = 0;
    fence_mbar_init();
  }
  if (warp == 9) {
    tmem_alloc<1>(smem_u32(tmem_slot), 512);
    tmem_relinquish<1>();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(tmem_slot);

  if (warp == 8) {
    if (lane == 0 && n_blocks > 0) {
      // ------------------------------------------------------------------ copies
      mbar_expect_tx(bar(Q_FULL), C::Q_BYTES);
      for (int kc = 0; kc < 4; ++kc) tma_load_3d(sQ + kc * (TT * 128), &p.tmQ, bar(Q_FULL), p.q_col0 + h * HD + kc * 64, q0, b);
      bool ok = true;
      int slot = 0, n = 0;
      auto load = [&](const void* map, int col0, int j) {              // a tile as two halves of 128 columns
        for (int c = 0; c < 2 && ok; ++c, ++n) {
          if (n >= C::SLOTS) ok = mbar_wait(bar(EMPTY + slot), (n / C::SLOTS - 1) & 1, abort_smem, p.status, SITE_SMEM_EMPTY);
          if (!ok) return;
          mbar_expect_tx(bar(FULL + slot), C::SLOT);
          for (int kc = 0; kc < 2; ++kc)
            tma_load_3d(ring + slot * C::SLOT + kc * (TT * 128), map, bar(FULL + slot), col0 + c * 128 + kc * 64, (j0 + j) * TT, b);
          if (++slot == C::SLOTS) slot = 0;
        }
      };
      load(&p.tmK, p.k_col0 + hk * HD, 0);
      for (int j = 0; ok && j < n_blocks; ++j) {
        if (j + 1 < n_blocks) load(&p.tmK, p.k_col0 + hk * HD, j + 1);
        if (ok) load(&p.tmV, p.v_col0 + hk * HD, j);
      }
    }
  } else if (warp == 9) {
    if (n_blocks > 0) {
      // ------------------------------------------------------------------ products (warp-uniform, one elected lane issues)
      constexpr uint32_t idesc_s = umma_idesc_bf16(TT, TT, 0, 0);
      constexpr uint32_t idesc_o = umma_idesc_bf16(TT, 128, 0, 1);           // half of the head dims; V is MN-major
      const bool leader = elect_one();
      const uint64_t dq0 = umma_smem_desc(sQ, 16, 1024), dk0 = umma_smem_desc(ring, 16, 1024), dv0 = umma_smem_desc(ring, TT * 128, 1024);
      int slot = 0, n = 0;
      bool ok = mbar_wait_warp(bar(Q_FULL), 0, abort_smem, p.status, SITE_SMEM_FULL);
      auto issue_s = [&](int j) {
        for (int c = 0; c < 2 && ok; ++c, ++n) {
          ok = mbar_wait_warp(bar(FULL + slot), (n / C::SLOTS) & 1, abort_smem, p.status, SITE_SMEM_FULL);
          if (!ok) return;
          tc_fence_after();
          const uint64_t da = dq0 + (uint32_t)(c * 2 * (TT * 128) / 16), db = dk0 + (uint32_t)(slot * (C::SLOT / 16));
          if (leader) {
#pragma unroll
            for (int k = 0; k < 8; ++k) {
              const int off = ((k / 4) * (TT * 128) + (k % 4) * 32) / 16;
              umma_f16<1>(tmem + (j & 1) * 128, da + off, db + off, idesc_s, (c | k) ? 1u : 0u);
            }
            umma_commit(bar(EMPTY + slot));
            if (c == 1) umma_commit(bar(S_FULL + (j & 1)));
          }
          __syncwarp();
          if (++slot == C::SLOTS) slot = 0;
        }
      };
      // the ring's order is K0 K1 V0 K2 V1 ..: V of block j lies before K of block j + 2
      if (ok) issue_s(0);
      if (ok && n_blocks > 1) issue_s(1);
      for (int j = 0; ok && j < n_blocks; ++j) {
        const int g = j & 1, s0 = slot, s1 = slot + 1 == C::SLOTS ? 0 : slot + 1;
        ok = mbar_wait_warp(bar(FULL + s0), (n / C::SLOTS) & 1, abort_smem, p.status, SITE_SMEM_FULL);
        if (ok) ok = mbar_wait_warp(bar(FULL + s1), ((n + 1) / C::SLOTS) & 1, abort_smem, p.status, SITE_SMEM_FULL);
        if (ok) ok = mbar_wait_warp(bar(P_HALF + g), (j >> 1) & 1, abort_smem, p.status, SITE_TMEM_FULL);
        if (!ok) break;
        tc_fence_after();
        const uint64_t db[2] = {dv0 + (uint32_t)(s0 * (C::SLOT / 16)), dv0 + (uint32_t)(s1 * (C::SLOT / 16))};
        const uint32_t first = j ? 1u : 0u;
        if (leader) {
#pragma unroll
          for (int k = 0; k < 4; ++k)
#pragma unroll
            for (int c = 0; c < 2; ++c)
              umma_f16_ts(tmem + C::O_COL0 + c * 128, tmem + g * 128 + k * 8, db[c] + k * 128, idesc_o, k ? 1u : first);
        }
        __syncwarp();
        ok = mbar_wait_warp(bar(P_FULL + g), (j >> 1) & 1, abort_smem, p.status, SITE_TMEM_FULL);
        if (!ok) break;
        tc_fence_after();
        if (leader) {
#pragma unroll
          for (int k = 4; k < 8; ++k)
#pragma unroll
            for (int c = 0; c < 2; ++c)
              umma_f16_ts(tmem + C::O_COL0 + c * 128, tmem + g * 128 + k * 8, db[c] + k * 128, idesc_o, 1u);
          umma_commit(bar(EMPTY + s0));
          umma_commit(bar(EMPTY + s1));
          umma_commit(bar(O_DONE + g));
        }
        __syncwarp();
        n += 2;
        slot = s1 + 1 == C::SLOTS ? 0 : s1 + 1;
        if (j + 2 < n_blocks) issue_s(j + 2);
      }
    }
  } else {
    // -------------------------------------------------------------------- softmax warps: thread = query row, every other block
    const int g = warp >> 2;
    const int row = threadIdx.x & 127;                 // == TMEM lane
    const int qi = q0 + row;
    const int qpos = p.q_off + qi * p.q_stride;
    const uint32_t lane_addr = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    const uint32_t s_addr = lane_addr + g * 128, o_addr = lane_addr + C::O_COL0;
    int k_first = 0, k_end = p.Tk;                     // keys this row sees: indices [k_first, k_end)
    if (p.causal) k_end = min(k_end, floor_div(qpos - p.k_off, p.k_stride) + 1);
    if (p.window > 0) k_first = max(0, floor_div(qpos - p.window - p.k_off, p.k_stride) + 1);
    int full_lo = 0, full_hi = p.Tk;                   // a block that every row sees whole needs no mask
    if (p.causal) full_hi = min(full_hi, floor_div(p.q_off + q0 * p.q_stride - p.k_off, p.k_stride) + 1);
    if (p.window > 0) full_lo = max(0, floor_div(p.q_off + (q0 + TT - 1) * p.q_stride - p.window - p.k_off, p.k_stride) + 1);
    const float thr = 8.f / p.scale_log2;              // the reference point moves when the max grew by > 2^8
    float m_at = -CUDART_INF_F, l = 0.f;               // own row sum, relative to the point it was last brought to
    DropoutRow dr;
    bool ok = true;
    for (int j = g; j < n_blocks; j += 2) {
      ok = mbar_wait(bar(S_FULL + g), (j >> 1) & 1, abort_smem, p.status, SITE_TMEM_FULL);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      uint32_t r[4][32];
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld_32x32(s_addr + c * 32, r[c]);
      tmem_ld_wait();
      const int kbase = (j0 + j) * TT;
      if (kbase < full_lo || kbase + TT > full_hi) {
        const int first = k_first - kbase, end = k_end - kbase;
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (c * 32 + i < first || c * 32 + i >= end) r[c][i] = 0xff800000u;     // -inf: exp2 gives an exact zero
      }
      float mxs[4] = {-CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F};
#pragma unroll
      for (int i = 0; i < 32; ++i)
#pragma unroll
        for (int c = 0; c < 4; ++c) mxs[c] = fmaxf(mxs[c], __uint_as_float(r[c][i]));
      const float mx = fmaxf(fmaxf(mxs[0], mxs[1]), fmaxf(mxs[2], mxs[3]));
      // the point the other group left for the block before
      float m_ref = -CUDART_INF_F;
      if (j > 0) {
        ok = mbar_wait(bar(M_READY + (g ^ 1)), ((j - 1) >> 1) & 1, abort_smem, p.status, SITE_SMEM_FULL);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        m_ref = m_s[(g ^ 1) * TT + row];
      }
      float alpha = 1.f;
      if (mx > m_ref + thr) {                          // also the first block with a visible key (m_ref = -inf)
        alpha = ex2_approx((m_ref - mx) * p.scale_log2);          // ex2(-inf) = 0
        m_ref = mx;
      }
      m_s[g * TT + row] = m_ref;
      mbar_arrive(bar(M_READY + g));
      // tcgen05.ld / .st are warp-collective: the decision must be the same for all 32 rows of a warp.  Never for the
      // first block: its product overwrites O.
      if (j > 0 && __any_sync(0xffffffffu, alpha != 1.f)) {
        ok = mbar_wait(bar(O_DONE + (g ^ 1)), ((j - 1) >> 1) & 1, abort_smem, p.status, SITE_TMEM_EMPTY);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
#pragma unroll 1
        for (int c = 0; c < HD / 16; ++c) {
          uint32_t o[16];
          tmem_ld_32x16(o_addr + c * 16, o);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
          tmem_st_32x16(o_addr + c * 16, o);
        }
      }
      const float neg_ms = (m_ref == -CUDART_INF_F) ? 0.f : -m_ref * p.scale_log2;
      if (m_at != m_ref) {
        l *= ex2_approx((m_at - m_ref) * p.scale_log2);
        m_at = m_ref;
      }
      if (DROP) dr.begin((uint32_t)(b * p.heads_total + p.head_off + h), (uint32_t)qpos);
      const F2 scale2 = f2(p.scale_log2, p.scale_log2), off2 = f2(neg_ms, neg_ms);
      F2 sum2[2] = {f2(0.f, 0.f), f2(0.f, 0.f)};
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t w[16];
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          float x0, x1;
          unpack(fma2(f2(__uint_as_float(r[c][i]), __uint_as_float(r[c][i + 1])), scale2, off2), x0, x1);
          float p0 = ex2_approx(x0), p1 = ex2_approx(x1);
          sum2[(i / 2) & 1] = add2(sum2[(i / 2) & 1], f2(p0, p1));      // the row sum is that of the undropped probabilities
          if (DROP) {
            const uint32_t kpos = (uint32_t)(p.k_off + (kbase + c * 32 + i) * p.k_stride);
            p0 = dr.keep(p.drop, kpos) ? p0 * p.drop.inv_keep : 0.f;
            p1 = dr.keep(p.drop, kpos + (uint32_t)p.k_stride) ? p1 * p.drop.inv_keep : 0.f;
          }
          __nv_bfloat162 hb = __floats2bfloat162_rn(p0, p1);
          w[i / 2] = *reinterpret_cast<uint32_t*>(&hb);
        }
        tmem_st_32x16(s_addr + c * 16, w);             // every score of the row is in registers by now
        if (c == 1 || c == 3) {
          tmem_st_wait();
          tc_fence_before();
          mbar_arrive(bar((c == 1 ? P_HALF : P_FULL) + g));
        }
      }
      float s0, s1;
      unpack(add2(sum2[0], sum2[1]), s0, s1);
      l += s0 + s1;
    }
    // ---- epilogue: O / l -> bf16 rows (half of the columns per group), log-sum-exp
    // The group of the last block waits for its product (it knows that the one before on this barrier is done: its scores
    // came later) and lets the other one go on at the bar.sync.  By then every M_READY has been waited for except the last
    // block's, whose reader would be the block after it: the points and the sums of both groups meet here.
    if (ok && n_blocks > 0 && g == ((n_blocks - 1) & 1))
      ok = mbar_wait(bar(O_DONE + g), ((n_blocks - 1) >> 1) & 1, abort_smem, p.status, SITE_TMEM_FULL);
    asm volatile("bar.sync 1, %0;" ::"n"(SM_THREADS) : "memory");
    tc_fence_after();
    m_s[g * TT + row] = m_at;
    l_s[g * TT + row] = l;
    asm volatile("bar.sync 1, %0;" ::"n"(SM_THREADS) : "memory");
    const float m_other = m_s[(g ^ 1) * TT + row], l_other = l_s[(g ^ 1) * TT + row];
    const float m_fin = fmaxf(m_at, m_other);
    float total = 0.f;
    if (m_fin != -CUDART_INF_F)
      total = l * ex2_approx((m_at - m_fin) * p.scale_log2) + l_other * ex2_approx((m_other - m_fin) * p.scale_log2);
    ok = __all_sync(0xffffffffu, ok);                  // the TMEM loads below are warp-collective: every lane takes part,
    if (ok) {                                          // only the global stores are predicated on the row being real
      const float inv = total > 0.f ? 1.f / total : 0.f;
      __nv_bfloat16* dst = p.out + ((long long)b * p.Tq + qi) * p.ldo + h * HD + g * 128;
#pragma unroll 1
      for (int c = 0; c < 4; ++c) {
        uint32_t o[32];
        if (n_blocks > 0) {
          tmem_ld_32x32(o_addr + g * 128 + c * 32, o);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) o[i] = 0;
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          uint4 q4;
          __nv_bfloat162* hb = reinterpret_cast<__nv_bfloat162*>(&q4);
#pragma unroll
          for (int i = 0; i < 4; ++i)
            hb[i] = __floats2bfloat162_rn(__uint_as_float(o[8 * q + 2 * i]) * inv, __uint_as_float(o[8 * q + 2 * i + 1]) * inv);
          if (qi < p.Tq) *reinterpret_cast<uint4*>(dst + c * 32 + q * 8) = q4;
        }
        __syncwarp();
      }
      if (p.lse && qi < p.Tq && g == 0)
        p.lse[((long long)b * p.H + h) * p.Tq + qi] =
            total > 0.f ? (m_fin * p.scale_log2 + log2f(total)) * 0.6931471805599453f : -CUDART_INF_F;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 9) {
    tc_fence_after();
    tmem_dealloc<1>(tmem, 512);
  }
}

// [sample][row][column]: what a tile reads past the last row of its sample is zero, not the next sample's.  (Hidden keys have
// P = 0, but 0 * NaN is NaN: a sample with NaN or infinities would reach the one before it.)
static bool map3d(CUtensorMap* tm, const void* base, uint64_t cols, uint64_t rows, uint64_t samples, uint64_t ld) {
  cuuint64_t dims[3] = {cols, rows, samples};
  cuuint64_t strides[2] = {ld * 2, rows * ld * 2};
  cuuint32_t box[3] = {64, TT, 1};
  cuuint32_t es[3] = {1, 1, 1};
  return encode_tiled(tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, base, dims, strides, box, es, CU_TENSOR_MAP_SWIZZLE_128B);
}

static bool map2d(CUtensorMap* tm, const void* base, uint64_t cols, uint64_t rows, uint64_t ld) {
  cuuint64_t dims[2] = {cols, rows};
  cuuint64_t strides[1] = {ld * 2};
  cuuint32_t box[2] = {64, TT};
  cuuint32_t es[2] = {1, 1};
  return encode_tiled(tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, base, dims, strides, box, es, CU_TENSOR_MAP_SWIZZLE_128B);
}

template <int HD>
static int launch(const MeshFlashArgs* a, cudaStream_t stream) {
  Params p;
  memset(&p, 0, sizeof(p));
  if (!map3d(&p.tmQ, a->q, (uint64_t)a->q_cols, (uint64_t)a->Tq, (uint64_t)a->B, (uint64_t)a->ldq)) return last_error_code();
  if (!map3d(&p.tmK, a->k, (uint64_t)a->k_cols, (uint64_t)a->Tk, (uint64_t)a->B, (uint64_t)a->ldk)) return last_error_code();
  if (!map3d(&p.tmV, a->v, (uint64_t)a->v_cols, (uint64_t)a->Tk, (uint64_t)a->B, (uint64_t)a->ldv)) return last_error_code();
  if (HD <= 128 && !(map2d(&p.tmK2, a->k, (uint64_t)a->k_cols, (uint64_t)a->B * a->Tk, (uint64_t)a->ldk) &&
                     map2d(&p.tmV2, a->v, (uint64_t)a->v_cols, (uint64_t)a->B * a->Tk, (uint64_t)a->ldv)))
    return last_error_code();
  p.out = (__nv_bfloat16*)a->out; p.ldo = a->ldo; p.lse = a->lse;
  p.B = a->B; p.H = a->H; p.Hkv = a->Hkv; p.Tq = a->Tq; p.Tk = a->Tk;
  p.q_col0 = a->q_col0; p.k_col0 = a->k_col0; p.v_col0 = a->v_col0;
  p.causal = a->causal; p.window = a->window;
  p.q_off = a->q_off; p.q_stride = a->q_stride > 0 ? a->q_stride : 1;
  p.k_off = a->k_off; p.k_stride = a->k_stride > 0 ? a->k_stride : 1;
  p.scale_log2 = a->scale * 1.4426950408889634f;
  p.status = (Status*)a->status;
  p.drop.p = a->dropout_p > 0.f ? a->dropout_p : 0.f;
  p.drop.inv_keep = p.drop.p > 0.f ? 1.f / (1.f - p.drop.p) : 1.f;
  p.drop.k0 = (uint32_t)(a->seed & 0xffffffffull) ^ (a->execution * 0x9E3779B9u);
  p.drop.k1 = (uint32_t)(a->seed >> 32);
  p.drop.site = a->site;
  p.head_off = a->head_off; p.heads_total = a->heads_total > 0 ? a->heads_total : a->H;
  if constexpr (HD <= 128) {
    auto kern = p.drop.p > 0.f ? flash_fwd2_kernel<HD, true> : flash_fwd2_kernel<HD, false>;
    static bool configured[2] = {false, false};
    if (!configured[p.drop.p > 0.f]) {
      MESH_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg2<HD>::SMEM));
      configured[p.drop.p > 0.f] = true;
    }
    dim3 grid(a->H * a->B, (a->Tq + 2 * TT - 1) / (2 * TT));
    kern<<<grid, THREADS2, Cfg2<HD>::SMEM, stream>>>(p);
  } else {
    auto kern = p.drop.p > 0.f ? flash_fwd256_kernel<true> : flash_fwd256_kernel<false>;
    static bool configured[2] = {false, false};
    if (!configured[p.drop.p > 0.f]) {
      MESH_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg256::SMEM));
      configured[p.drop.p > 0.f] = true;
    }
    dim3 grid(a->H * a->B, (a->Tq + TT - 1) / TT);
    kern<<<grid, THREADS2, Cfg256::SMEM, stream>>>(p);
  }
  MESH_CUDA_OK(cudaGetLastError());
  return 0;
}

}  // namespace fa
}  // namespace mesh

extern "C" int mesh_flash_attention_fwd(const MeshFlashArgs* a, void* stream) {
  using namespace mesh;
  if (a->H % a->Hkv) return set_error(-2, "flash_attention: query heads must be a multiple of KV heads");
  if (a->ldq % 8 || a->ldk % 8 || a->ldv % 8 || a->ldo % 8 || a->q_col0 % 8 || a->k_col0 % 8 || a->v_col0 % 8)
    return set_error(-2, "flash_attention: leading dimensions and head offsets must be multiples of 8 elements");
  if (a->Tq % 1 || a->B < 1) return set_error(-2, "flash_attention: empty problem");
  if (!(a->dropout_p >= 0.f && a->dropout_p < 1.f)) return set_error(-2, "flash_attention: dropout_p must be in [0, 1)");
  switch (a->head_dim) {
    case 64: return fa::launch<64>(a, (cudaStream_t)stream);
    case 128: return fa::launch<128>(a, (cudaStream_t)stream);
    case 256: return fa::launch<256>(a, (cudaStream_t)stream);
    default: return set_error(-2, "flash_attention: head_dim must be 64, 128 or 256");
  }
}
