// Flash attention backward on tcgen05 / TMEM: a serial kernel (dropout) and a pipelined one (everything else).
//
// One CTA owns one block of 128 keys of one KV head and walks the query blocks (of every query head of
// the group) that can see it.  Per query block, five tensor-core products run from the same shared-memory
// tiles, with no transposed copies — a transposed operand is the same bytes read through an MN-major
// descriptor:
//     S  = Q K^T            dP = dO V^T                      (accumulators in TMEM, one row per thread)
//     P  = exp(S*scale - L)  dS = P o (dP - Delta) * scale   (threads, written to shared memory as bf16)
//     dV += P^T dO          dK += dS^T Q                     (accumulate in TMEM across all query blocks)
//     dQ  = dS K            -> added to a float accumulator in global memory (several key blocks add to it)
// L is the log-sum-exp of the forward pass and Delta = rowsum(dO o O).  With the global L of a ring
// attention the same kernel yields each KV chunk's contribution (chunks are visited one at a time by
// the caller), masks are evaluated on logical positions exactly as in the forward kernel.
// Reference semantics: the backward of the blockwise attention of compiler/mesh_compiler/operations.py:7081-7166.
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
namespace fab {

constexpr int BQ = 128, BKV = 128;
constexpr int SM_THREADS = 256;       // 8 softmax warps: threads r and r + 128 share row r, half of the columns each
constexpr int THREADS = 288;          // + 1 copy/MMA warp

struct Params {
  CUtensorMap tmQ, tmK, tmV, tmdO;           // [sample][row][column], boxes of 64 columns and 128 rows
  CUtensorMap tmdQ;                          // fp32 [B][Tq][H*hd], box {32, 32, 1}
  const float* lse; const float* delta;      // [B, H, Tq]
  float* dq;                                 // fp32 [B*Tq, H*hd], zeroed by the caller
  __nv_bfloat16* dk; __nv_bfloat16* dv;      // [B*Tk, Hkv*hd] (bf16, written) ...
  float* dk_acc; float* dv_acc;              // ... or fp32 accumulators that are added to (ring attention)
  long long ld_dq, ld_dkv;
  int B, H, Hkv, Tq, Tk;
  int q_col0, k_col0, v_col0, do_col0;
  int causal, window, q_off, q_stride, k_off, k_stride;
  float scale, scale_log2;
  Status* status;
  DropoutKey drop;
  int head_off, heads_total;
};

__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ void tmem_ld32(uint32_t addr, uint32_t (&r)[32]) {
  tmem_ld_32x32(addr, r);
  tmem_ld_wait();
}

// bf16 row piece (32 columns) into the [kv/64][128 rows][128 B] swizzled tile
__device__ __forceinline__ void store_row32(uint32_t tile, int row, int c, const uint32_t (&w)[16]) {
  const uint32_t row_base = tile + (c / 2) * (128 * 128) + row * 128;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const uint32_t chunk = ((c & 1) * 4 + j) ^ (row & 7);
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(row_base + (chunk << 4)), "r"(w[4 * j]), "r"(w[4 * j + 1]),
                 "r"(w[4 * j + 2]), "r"(w[4 * j + 3]) : "memory");
  }
}

// dV and dK of one key row (thread = row, half of the head dimension) from tensor memory: bf16 outputs, or added to the
// fp32 accumulators.  The TMEM loads are warp-collective: only the stores are predicated on the row being real.
template <int HD>
__device__ __forceinline__ void write_dkv(const Params& p, uint32_t dv_addr, uint32_t dk_addr, int b, int hk, int kj, int half) {
  const long long off = ((long long)b * p.Tk + kj) * p.ld_dkv + hk * HD + half * (HD / 2);
#pragma unroll 1
  for (int which = 0; which < 2; ++which) {
    const uint32_t addr = (which ? dk_addr : dv_addr) + half * (HD / 2);
#pragma unroll 1
    for (int c = 0; c < HD / 64; ++c) {
      uint32_t r[32];
      tmem_ld32(addr + c * 32, r);
      if (kj < p.Tk && p.dk_acc) {
        float* dst = (which ? p.dk_acc : p.dv_acc) + off + c * 32;
#pragma unroll
        for (int e = 0; e < 32; e += 4) {
          float4 cur = *reinterpret_cast<float4*>(dst + e);
          cur.x += __uint_as_float(r[e]); cur.y += __uint_as_float(r[e + 1]);
          cur.z += __uint_as_float(r[e + 2]); cur.w += __uint_as_float(r[e + 3]);
          *reinterpret_cast<float4*>(dst + e) = cur;
        }
      } else if (kj < p.Tk) {
        __nv_bfloat16* dst = (which ? p.dk : p.dv) + off + c * 32;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          uint4 o;
          __nv_bfloat162* hb = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
          for (int e = 0; e < 4; ++e)
            hb[e] = __floats2bfloat162_rn(__uint_as_float(r[8 * j + 2 * e]), __uint_as_float(r[8 * j + 2 * e + 1]));
          *reinterpret_cast<uint4*>(dst + j * 8) = o;
        }
      }
      __syncwarp();
    }
  }
}

// nothing sees this key block: its gradients are zero
template <int HD>
__device__ __forceinline__ void zero_dkv(const Params& p, int b, int hk, int kj) {
  if (kj >= p.Tk) return;
  const long long off = ((long long)b * p.Tk + kj) * p.ld_dkv + hk * HD;
  for (int e = 0; e < HD; e += 8) {
    *reinterpret_cast<uint4*>(p.dk + off + e) = make_uint4(0, 0, 0, 0);
    *reinterpret_cast<uint4*>(p.dv + off + e) = make_uint4(0, 0, 0, 0);
  }
}

template <int HD>
__global__ void __launch_bounds__(THREADS, 1) flash_bwd_kernel(const __grid_constant__ Params p) {
  constexpr int KC = HD / 64;
  constexpr int TILE = 128 * HD * 2;          // Q, dO, K, V tiles
  constexpr int PT = 128 * 128 * 2;           // P, dS tiles
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t sK = base, sV = sK + TILE, sQ = sV + TILE, sdO = sQ + TILE, sP = sdO + TILE, sdS = sP + PT;
  const uint32_t bars = sdS + PT;
  auto bar = [&](int i) { return bars + 8u * i; };
  constexpr int KV_FULL = 0, Q_FULL = 1, SDP_FULL = 2, PDS_FULL = 3, MMA2_DONE = 4, DQ_READ = 5;
  uint8_t* gen = smem_raw + (base - smem_u32(smem_raw));
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(gen + 4 * TILE + 2 * PT + 8 * 8);
  volatile int* abort_smem = reinterpret_cast<volatile int*>(tmem_slot + 1);
  // TMEM columns: S / dQ at 0, dP at 128, dV at 256, dK at 256 + HD
  constexpr int C_S = 0, C_DP = 128, C_DV = 256, C_DK = 256 + HD;
  static_assert(C_DK + HD <= 512, "head_dim up to 128 fits tensor memory");

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int jb = blockIdx.x, hk = blockIdx.y, b = blockIdx.z;
  const int group = p.H / p.Hkv;
  const int k0 = jb * BKV;

  // query blocks that can see this key block
  const int kpos_lo = p.k_off + k0 * p.k_stride;
  const int kpos_hi = p.k_off + (min(k0 + BKV, p.Tk) - 1) * p.k_stride;
  int i_lo = 0, i_hi = (p.Tq + BQ - 1) / BQ;
  if (p.causal) {
    // queries with q_pos >= kpos_lo
    const int qmin = kpos_lo - p.q_off <= 0 ? 0 : (kpos_lo - p.q_off + p.q_stride - 1) / p.q_stride;
    i_lo = max(i_lo, qmin / BQ);
  }
  if (p.window > 0) {
    // queries with q_pos < kpos_hi + window
    const int qmax_pos = kpos_hi + p.window - 1;
    const int qmax = qmax_pos - p.q_off < 0 ? -1 : (qmax_pos - p.q_off) / p.q_stride;
    i_hi = min(i_hi, qmax / BQ + 1);
    if (qmax < 0) i_hi = 0;
  }
  const int n_q = max(0, i_hi - i_lo);
  const int n_iter = n_q * group;

  if (threadIdx.x == 0) {
    mbar_init(bar(KV_FULL), 1);
    mbar_init(bar(Q_FULL), 1);
    mbar_init(bar(SDP_FULL), 1);
    mbar_init(bar(PDS_FULL), SM_THREADS);
    mbar_init(bar(MMA2_DONE), 1);
    mbar_init(bar(DQ_READ), SM_THREADS);
    *abort_smem = 0;
    fence_mbar_init();
  }
  if (warp == 8) {
    tmem_alloc<1>(smem_u32(tmem_slot), 512);
    tmem_relinquish<1>();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(tmem_slot);

  if (warp == 8) {
    if (lane == 0 && n_iter > 0) {
      mbar_expect_tx(bar(KV_FULL), 2 * TILE);
      for (int kc = 0; kc < KC; ++kc) {
        tma_load_3d(sK + kc * (128 * 128), &p.tmK, bar(KV_FULL), p.k_col0 + hk * HD + kc * 64, k0, b);
        tma_load_3d(sV + kc * (128 * 128), &p.tmV, bar(KV_FULL), p.v_col0 + hk * HD + kc * 64, k0, b);
      }
      constexpr uint32_t id_s = umma_idesc_bf16(128, 128, 0, 0);        // Q K^T and dO V^T: both K-major over head_dim
      constexpr uint32_t id_t = umma_idesc_bf16(128, HD, 1, 1);         // P^T dO and dS^T Q: A and B MN-major, K = queries
      constexpr uint32_t id_q = umma_idesc_bf16(128, HD, 0, 1);         // dS K: A K-major over keys, B = K MN-major
      bool ok = mbar_wait(bar(KV_FULL), 0, abort_smem, p.status, SITE_SMEM_FULL);
      for (int it = 0; ok && it < n_iter; ++it) {
        const int g = it / n_q, i = i_lo + it % n_q;
        const int h = hk * group + g;
        // Q and dO of this block may be overwritten once the second group of products of the previous iteration is done
        if (it > 0) {
          ok = mbar_wait(bar(MMA2_DONE), (it - 1) & 1, abort_smem, p.status, SITE_SMEM_EMPTY);
          if (!ok) break;
        }
        mbar_expect_tx(bar(Q_FULL), 2 * TILE);
        for (int kc = 0; kc < KC; ++kc) {
          tma_load_3d(sQ + kc * (128 * 128), &p.tmQ, bar(Q_FULL), p.q_col0 + h * HD + kc * 64, i * BQ, b);
          tma_load_3d(sdO + kc * (128 * 128), &p.tmdO, bar(Q_FULL), p.do_col0 + h * HD + kc * 64, i * BQ, b);
        }
        ok = mbar_wait(bar(Q_FULL), it & 1, abort_smem, p.status, SITE_SMEM_FULL);
        if (!ok) break;
        // the S / dQ columns are free once the threads have read dQ of the previous iteration
        if (it > 0) {
          ok = mbar_wait(bar(DQ_READ), (it - 1) & 1, abort_smem, p.status, SITE_TMEM_EMPTY);
          if (!ok) break;
        }
        tc_fence_after();
#pragma unroll
        for (int kc = 0; kc < KC; ++kc)
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const uint32_t off = kc * (128 * 128) + k * 32;
            umma_f16<1>(tmem + C_S, umma_smem_desc(sQ + off, 16, 1024), umma_smem_desc(sK + off, 16, 1024), id_s, (kc | k) ? 1u : 0u);
            umma_f16<1>(tmem + C_DP, umma_smem_desc(sdO + off, 16, 1024), umma_smem_desc(sV + off, 16, 1024), id_s, (kc | k) ? 1u : 0u);
          }
        umma_commit(bar(SDP_FULL));
        // second group: needs P and dS from the threads
        ok = mbar_wait(bar(PDS_FULL), it & 1, abort_smem, p.status, SITE_TMEM_FULL);
        if (!ok) break;
        tc_fence_after();
#pragma unroll
        for (int k = 0; k < 128 / 16; ++k) {
          // transposed reads: MN = keys (groups of 64, one [128 rows][128 B] slab apart), K = the 128 query rows
          const uint64_t a_pt = umma_smem_desc(sP + k * 2048, 128 * 128, 1024);
          const uint64_t a_dst = umma_smem_desc(sdS + k * 2048, 128 * 128, 1024);
          const uint64_t b_do = umma_smem_desc(sdO + k * 2048, 128 * 128, 1024);
          const uint64_t b_q = umma_smem_desc(sQ + k * 2048, 128 * 128, 1024);
          umma_f16<1>(tmem + C_DV, a_pt, b_do, id_t, (it | k) ? 1u : 0u);
          umma_f16<1>(tmem + C_DK, a_dst, b_q, id_t, (it | k) ? 1u : 0u);
          // dQ = dS K: A = dS as written (K-major over the keys), B = K tile read MN-major
          const uint64_t a_ds = umma_smem_desc(sdS + (k / 4) * (128 * 128) + (k % 4) * 32, 16, 1024);
          const uint64_t b_k = umma_smem_desc(sK + k * 2048, 128 * 128, 1024);
          umma_f16<1>(tmem + C_S, a_ds, b_k, id_q, k ? 1u : 0u);
        }
        umma_commit(bar(MMA2_DONE));
      }
    }
  } else {
    const int row = threadIdx.x & 127;                // == TMEM lane; query row in the loop, key row at the end
    const int half = threadIdx.x >> 7;                // which 64 key columns of S / dP, which half of the dQ/dK/dV columns
    const uint32_t lane_addr = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    bool ok = true;
    for (int it = 0; ok && it < n_iter; ++it) {
      const int g = it / n_q, i = i_lo + it % n_q;
      const int h = hk * group + g;
      const int qi = i * BQ + row;
      const int qpos = p.q_off + qi * p.q_stride;
      const bool qreal = qi < p.Tq;
      const float L = qreal ? p.lse[((long long)b * p.H + h) * p.Tq + qi] : -CUDART_INF_F;
      const float dl = qreal ? p.delta[((long long)b * p.H + h) * p.Tq + qi] : 0.f;
      // rows with no visible key at all (L = -inf) and rows past the end get P = 0 through an infinite offset
      const float negL2 = (L == -CUDART_INF_F) ? -CUDART_INF_F : -L * 1.4426950408889634f;
      // does a mask or the end of the keys / queries cut into this (query block, key block) pair?
      const int qpos_lo = p.q_off + i * BQ * p.q_stride, qpos_hi = p.q_off + (i * BQ + BQ - 1) * p.q_stride;
      const bool masked = (k0 + BKV > p.Tk) || (p.causal && kpos_hi > qpos_lo) ||
                          (p.window > 0 && kpos_lo <= qpos_hi - p.window);
      ok = mbar_wait(bar(SDP_FULL), it & 1, abort_smem, p.status, SITE_TMEM_FULL);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      // P and dS may be overwritten: SDP_FULL of this iteration was issued after the MMA warp had waited for the
      // previous iteration's second group of products, which read them
      DropoutRow dr;
      if (p.drop.p > 0.f) dr.begin((uint32_t)(b * p.heads_total + p.head_off + h), (uint32_t)qpos);
#pragma unroll 1
      for (int c = 0; c < 2; ++c) {
        uint32_t rs[32], rp[32];
        tmem_ld_32x32(lane_addr + C_S + half * 64 + c * 32, rs);
        tmem_ld_32x32(lane_addr + C_DP + half * 64 + c * 32, rp);
        tmem_ld_wait();
        uint32_t wp[16], wd[16];
#pragma unroll
        for (int e = 0; e < 32; e += 2) {
          float pv[2], dv[2];
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            float pr = ex2_approx(fmaf(__uint_as_float(rs[e + u]), p.scale_log2, negL2));
            if (masked) {
              const int kj = k0 + half * 64 + c * 32 + e + u;
              const int kpos = p.k_off + kj * p.k_stride;
              const bool vis = kj < p.Tk && (!p.causal || kpos <= qpos) && (p.window <= 0 || kpos > qpos - p.window);
              pr = vis ? pr : 0.f;
            }
            // dropout: dV sees the dropped, rescaled probabilities; dP comes back through the same mask
            float m = 1.f;
            if (p.drop.p > 0.f) {
              const uint32_t kpos = (uint32_t)(p.k_off + (k0 + half * 64 + c * 32 + e + u) * p.k_stride);
              m = dr.keep(p.drop, kpos) ? p.drop.inv_keep : 0.f;
            }
            pv[u] = pr * m;
            dv[u] = pr * (__uint_as_float(rp[e + u]) * m - dl) * p.scale;
          }
          __nv_bfloat162 hp = __floats2bfloat162_rn(pv[0], pv[1]);
          __nv_bfloat162 hd2 = __floats2bfloat162_rn(dv[0], dv[1]);
          wp[e / 2] = *reinterpret_cast<uint32_t*>(&hp);
          wd[e / 2] = *reinterpret_cast<uint32_t*>(&hd2);
        }
        store_row32(sP, row, half * 2 + c, wp);
        store_row32(sdS, row, half * 2 + c, wd);
      }
      fence_proxy_async_smem();
      tc_fence_before();
      mbar_arrive(bar(PDS_FULL));
      // dQ tile of this (query block, key block): add this thread's half of the row into the float accumulator
      ok = mbar_wait(bar(MMA2_DONE), it & 1, abort_smem, p.status, SITE_TMEM_FULL);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      float* dq = p.dq + ((long long)b * p.Tq + qi) * p.ld_dq + h * HD + half * (HD / 2);
#pragma unroll 1
      for (int c = 0; c < HD / 64; ++c) {
        uint32_t r[32];
        tmem_ld32(lane_addr + C_S + half * (HD / 2) + c * 32, r);
        if (qreal) {
#pragma unroll
          for (int e = 0; e < 32; e += 4)
            asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dq + c * 32 + e), "f"(__uint_as_float(r[e])),
                         "f"(__uint_as_float(r[e + 1])), "f"(__uint_as_float(r[e + 2])), "f"(__uint_as_float(r[e + 3])) : "memory");
        }
      }
      tc_fence_before();
      mbar_arrive(bar(DQ_READ));
    }
    // ---- dK, dV of this key block (thread = key row, half of the head dimension)
    ok = __all_sync(0xffffffffu, ok);
    if (ok && n_iter > 0) write_dkv<HD>(p, lane_addr + C_DV, lane_addr + C_DK, b, hk, k0 + row, half);
    else if (n_iter == 0 && !p.dk_acc && half == 0) zero_dkv<HD>(p, b, hk, k0 + row);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 8) {
    tc_fence_after();
    tmem_dealloc<1>(tmem, 512);
  }
}

// ------------------------------------------------------------------------------------------------ pipelined backward
// Without dropout.  As above one CTA owns 128 keys of a KV head and walks the query blocks that see them, but the scores
// are computed transposed (rows = keys) and the five products of consecutive query blocks overlap with the threads:
//
//     tensor core   ... dV += P^T dO | S' = K Q'^T | dQ = dS K | dK += dS^T Q | dP' = V dO'^T ...     (' = next block)
//     warps 0-7     P from S, dS from P and dP: a thread holds one key row and half of the query columns
//     warps 8-11    add dQ of the block to the float accumulator while dK runs: 32 x 32 pieces through shared memory
//                   and one reducing bulk copy each.  (Reductions straight from registers, red.global.add.v2 with four
//                   lanes on a 32-byte sector, held the whole pipeline up: 942 us instead of 706 us then, at one sequence of
//                   8192, 16 heads of 128, causal.)
//     warp 12       copies: K, V once; Q, L and Delta of the query blocks through two stages, dO through one (it is
//                   free from dV of a block on and needed again three products later; the other 32 KB stage dQ)
//     warp 13       issues the products in the order above
//
// P^T goes back to tensor memory as bf16 over the columns of S that its thread has read, and feeds dV from there; only
// dS passes through shared memory, where dK reads it along the keys and dQ across them.  dQ takes the columns of dP,
// which every thread has read by the time dS is complete.
//
// Bound by the chain dP -> dS -> dQ -> drain -> dP' beside a tensor pipe that needs 2560 cycles per pair of blocks at
// head size 128.  Measured at one sequence of 8192, 16 heads of 128, causal: 1967 us with the serial kernel above,
// 694 us with this one (990 TFLOP/s); heads of 64: 477 us.  Dropout stays with the kernel above: there a thread holds
// a query row and pays one generator call for four keys, here it would pay one for every score.
constexpr int THREADS2 = 448;

struct Bars2 {
  static constexpr int KV_FULL = 0, Q_FULL = 1, Q_EMPTY = 3, DO_FULL = 5, DO_EMPTY = 6, S_FULL = 7, P_FULL = 8, DP_FULL = 9,
                       DS_FULL = 10, DQ_FULL = 11, DQ_READ = 12, ACC_DONE = 13, N = 14;
};

template <int HD>
struct Cfg2 {
  static constexpr int KC = HD / 64;
  static constexpr int TILE = 128 * HD * 2;            // K, V, Q, dO tiles
  static constexpr int PT = 128 * 128 * 2;             // dS tile
  static constexpr int ROWS = 2 * 2 * 128 * 4;         // L and Delta of two query blocks
  static constexpr int RED = 4 * 2 * 4096;             // two 32 x 32 fp32 pieces of dQ per warp
  static constexpr int SMEM = 5 * TILE + PT + RED + ROWS + 8 * Bars2::N + 16;    // no room to align by hand at 128
};

template <int HD>
__global__ void __launch_bounds__(THREADS2, 1) flash_bwd2_kernel(const __grid_constant__ Params p) {
  using C = Cfg2<HD>;
  using B_ = Bars2;
  constexpr int KC = C::KC, TILE = C::TILE;
  extern __shared__ __align__(1024) uint8_t smem_al[];
  const uint32_t base = smem_u32(smem_al);
  if (base & 1023u) {                                  // the swizzled tiles need it; nothing is placed before them
    if (threadIdx.x == 0) status_record(p.status, MESH_ALIGN, SITE_NONE, 1024, base);
    return;
  }
  const uint32_t sK = base, sV = sK + TILE, sQ = sV + TILE, sdO = sQ + 2 * TILE, sdS = sdO + TILE, sRed = sdS + C::PT;
  uint8_t* gen = smem_al;
  float* rows_s = reinterpret_cast<float*>(gen + 5 * TILE + C::PT + C::RED);   // [stage][-L * log2(e), -Delta * scale][128]
  const uint32_t bars = sRed + C::RED + C::ROWS;
  auto bar = [&](int i) { return bars + 8u * i; };
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(gen + 5 * TILE + C::PT + C::RED + C::ROWS + 8 * B_::N);
  volatile int* abort_smem = reinterpret_cast<volatile int*>(tmem_slot + 1);
  // tensor memory columns: S (P^T), dP (dQ), dV, dK
  constexpr int C_S = 0, C_DP = 128, C_DQ = 128, C_DV = 256, C_DK = 256 + HD;
  static_assert(C_DK + HD <= 512, "head_dim up to 128 fits tensor memory");

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // key blocks in the slow grid dimension: the first ones, which the causal mask hides from nobody, start first
  const int jb = blockIdx.y, hk = blockIdx.x % p.Hkv, b = blockIdx.x / p.Hkv;
  const int group = p.H / p.Hkv;
  const int k0 = jb * BKV;

  // query blocks that can see this key block
  const int kpos_lo = p.k_off + k0 * p.k_stride;
  const int kpos_hi = p.k_off + (min(k0 + BKV, p.Tk) - 1) * p.k_stride;
  int i_lo = 0, i_hi = (p.Tq + BQ - 1) / BQ;
  if (p.causal) {
    const int qmin = kpos_lo - p.q_off <= 0 ? 0 : (kpos_lo - p.q_off + p.q_stride - 1) / p.q_stride;
    i_lo = max(i_lo, qmin / BQ);
  }
  if (p.window > 0) {
    const int qmax_pos = kpos_hi + p.window - 1;
    const int qmax = qmax_pos - p.q_off < 0 ? -1 : (qmax_pos - p.q_off) / p.q_stride;
    i_hi = min(i_hi, qmax / BQ + 1);
    if (qmax < 0) i_hi = 0;
  }
  const int n_q = max(0, i_hi - i_lo);
  const int n_iter = n_q * group;

  if (threadIdx.x == 0) {
    mbar_init(bar(B_::KV_FULL), 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(bar(B_::Q_FULL + s), 1);
      mbar_init(bar(B_::Q_EMPTY + s), 1);
    }
    mbar_init(bar(B_::DO_FULL), 33);                   // the copy and 32 lanes that stored L and Delta
    mbar_init(bar(B_::DO_EMPTY), 1);
    mbar_init(bar(B_::S_FULL), 1);
    mbar_init(bar(B_::P_FULL), SM_THREADS);
    mbar_init(bar(B_::DP_FULL), 1);
    mbar_init(bar(B_::DS_FULL), SM_THREADS);
    mbar_init(bar(B_::DQ_FULL), 1);
    mbar_init(bar(B_::DQ_READ), 128);
    mbar_init(bar(B_::ACC_DONE), 1);
    *abort_smem = 0;
    fence_mbar_init();
  }
  if (warp == 13) {
    tmem_alloc<1>(smem_u32(tmem_slot), 512);
    tmem_relinquish<1>();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(tmem_slot);

  if (warp == 12) {
    // -------------------------------------------------------------------- copies
    if (n_iter > 0) {
      if (lane == 0) {
        mbar_expect_tx(bar(B_::KV_FULL), 2 * TILE);
        for (int kc = 0; kc < KC; ++kc) {
          tma_load_3d(sK + kc * (128 * 128), &p.tmK, bar(B_::KV_FULL), p.k_col0 + hk * HD + kc * 64, k0, b);
          tma_load_3d(sV + kc * (128 * 128), &p.tmV, bar(B_::KV_FULL), p.v_col0 + hk * HD + kc * 64, k0, b);
        }
      }
      bool ok = true;
      for (int it = 0; ok && it < n_iter; ++it) {
        const int s = it & 1;
        const int g = it / n_q, i = i_lo + it % n_q;
        const int h = hk * group + g;
        if (it >= 2) ok = mbar_wait(bar(B_::Q_EMPTY + s), ((it >> 1) - 1) & 1, abort_smem, p.status, SITE_SMEM_EMPTY);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        if (lane == 0) {
          mbar_expect_tx(bar(B_::Q_FULL + s), TILE);
          for (int kc = 0; kc < KC; ++kc)
            tma_load_3d(sQ + s * TILE + kc * (128 * 128), &p.tmQ, bar(B_::Q_FULL + s), p.q_col0 + h * HD + kc * 64, i * BQ, b);
        }
        if (it >= 1) ok = mbar_wait(bar(B_::DO_EMPTY), (it - 1) & 1, abort_smem, p.status, SITE_SMEM_EMPTY);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        if (lane == 0) {
          mbar_expect_tx(bar(B_::DO_FULL), TILE);
          for (int kc = 0; kc < KC; ++kc)
            tma_load_3d(sdO + kc * (128 * 128), &p.tmdO, bar(B_::DO_FULL), p.do_col0 + h * HD + kc * 64, i * BQ, b);
        }
        // rows with no visible key at all (L = -inf) and rows past the end get P = 0 through an infinite offset
        const long long row0 = ((long long)b * p.H + h) * p.Tq + i * BQ;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int r = u * 32 + lane;
          const bool real = i * BQ + r < p.Tq;
          const float L = real ? __ldg(p.lse + row0 + r) : -CUDART_INF_F;
          const float dl = real ? __ldg(p.delta + row0 + r) : 0.f;
          rows_s[s * 256 + r] = (L == -CUDART_INF_F) ? -CUDART_INF_F : -L * 1.4426950408889634f;
          rows_s[s * 256 + 128 + r] = -dl * p.scale;
        }
        mbar_arrive(bar(B_::DO_FULL));
      }
    }
  } else if (warp == 13) {
    if (n_iter > 0) {
      // ------------------------------------------------------------------ products: the whole warp runs the loop and one
      // elected lane issues, so that descriptors and addresses stay in uniform registers
      constexpr uint32_t id_s = umma_idesc_bf16(128, 128, 0, 0);        // K Q^T and V dO^T: both K-major over head_dim
      constexpr uint32_t id_t = umma_idesc_bf16(128, HD, 0, 1);         // P^T dO and dS^T Q: A along the queries, B MN-major
      constexpr uint32_t id_q = umma_idesc_bf16(128, HD, 1, 1);         // dS K: A read across the keys
      const bool leader = elect_one();
      // K-major and MN-major descriptors of the tiles; 16 deeper in k is 32 bytes in the one and 2 KiB in the other
      const uint64_t kK = umma_smem_desc(sK, 16, 1024), kV = umma_smem_desc(sV, 16, 1024), kQ = umma_smem_desc(sQ, 16, 1024);
      const uint64_t kdO = umma_smem_desc(sdO, 16, 1024), kdS = umma_smem_desc(sdS, 16, 1024);
      const uint64_t mK = umma_smem_desc(sK, 128 * 128, 1024), mQ = umma_smem_desc(sQ, 128 * 128, 1024);
      const uint64_t mdO = umma_smem_desc(sdO, 128 * 128, 1024), mdS = umma_smem_desc(sdS, 128 * 128, 1024);
      auto issue_nt = [&](uint32_t d, uint64_t a, uint64_t bm) {
#pragma unroll
        for (int kc = 0; kc < KC; ++kc)
#pragma unroll
          for (int k = 0; k < 4; ++k)
            umma_f16<1>(d, a + (kc * (128 * 128) + k * 32) / 16, bm + (kc * (128 * 128) + k * 32) / 16, id_s, (kc | k) ? 1u : 0u);
      };
      bool ok = mbar_wait_warp(bar(B_::KV_FULL), 0, abort_smem, p.status, SITE_SMEM_FULL);
      if (ok) ok = mbar_wait_warp(bar(B_::Q_FULL), 0, abort_smem, p.status, SITE_SMEM_FULL);
      if (ok) {
        tc_fence_after();
        if (leader) {
          issue_nt(tmem + C_S, kK, kQ);
          umma_commit(bar(B_::S_FULL));
        }
        ok = mbar_wait_warp(bar(B_::DO_FULL), 0, abort_smem, p.status, SITE_SMEM_FULL);
      }
      if (ok) {
        tc_fence_after();
        if (leader) {
          issue_nt(tmem + C_DP, kV, kdO);
          umma_commit(bar(B_::DP_FULL));
        }
      }
      for (int it = 0; ok && it < n_iter; ++it) {
        const int s = it & 1, sn = s ^ 1;
        const bool more = it + 1 < n_iter;
        const uint32_t first = it ? 1u : 0u;
        if (more) ok = mbar_wait_warp(bar(B_::Q_FULL + sn), ((it + 1) >> 1) & 1, abort_smem, p.status, SITE_SMEM_FULL);
        if (ok) ok = mbar_wait_warp(bar(B_::P_FULL), it & 1, abort_smem, p.status, SITE_TMEM_FULL);
        if (!ok) break;
        tc_fence_after();
        if (leader) {
#pragma unroll
          for (int k = 0; k < 8; ++k)                  // P^T: 64 queries in columns 0.., the others in columns 64..
            umma_f16_ts(tmem + C_DV, tmem + C_S + (k < 4 ? k * 8 : 64 + (k - 4) * 8), mdO + k * 128, id_t, k ? 1u : first);
          umma_commit(bar(B_::DO_EMPTY));
          if (more) {
            issue_nt(tmem + C_S, kK, kQ + (uint32_t)(sn * (TILE >> 4)));
            umma_commit(bar(B_::S_FULL));
          }
        }
        __syncwarp();
        ok = mbar_wait_warp(bar(B_::DS_FULL), it & 1, abort_smem, p.status, SITE_TMEM_FULL);
        if (!ok) break;
        tc_fence_after();
        if (leader) {
#pragma unroll
          for (int k = 0; k < 8; ++k) umma_f16<1>(tmem + C_DQ, mdS + k * 128, mK + k * 128, id_q, k ? 1u : 0u);
          umma_commit(bar(B_::DQ_FULL));
          const uint64_t q = mQ + (uint32_t)(s * (TILE >> 4));
#pragma unroll
          for (int k = 0; k < 8; ++k)
            umma_f16<1>(tmem + C_DK, kdS + ((k / 4) * (128 * 128) + (k % 4) * 32) / 16, q + k * 128, id_t, k ? 1u : first);
          umma_commit(bar(B_::Q_EMPTY + s));
        }
        __syncwarp();
        if (more) {
          ok = mbar_wait_warp(bar(B_::DO_FULL), (it + 1) & 1, abort_smem, p.status, SITE_SMEM_FULL);
          if (ok) ok = mbar_wait_warp(bar(B_::DQ_READ), it & 1, abort_smem, p.status, SITE_TMEM_EMPTY);
          if (!ok) break;
          tc_fence_after();
          if (leader) {
            issue_nt(tmem + C_DP, kV, kdO);
            umma_commit(bar(B_::DP_FULL));             // also: dK and dQ of this block are done with dS
          }
          __syncwarp();
        }
      }
      if (ok && leader) umma_commit(bar(B_::ACC_DONE));
    }
  } else if (warp >= 8) {
    // -------------------------------------------------------------------- dQ into the float accumulator
    const uint32_t lane_addr = tmem + ((uint32_t)((warp & 3) * 32) << 16) + C_DQ;
    const uint32_t stage = sRed + (warp & 3) * 8192;
    bool ok = true;
    for (int it = 0; it < n_iter; ++it) {
      const int g = it / n_q, i = i_lo + it % n_q;
      const int h = hk * group + g;
      ok = mbar_wait(bar(B_::DQ_FULL), it & 1, abort_smem, p.status, SITE_TMEM_FULL);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
#pragma unroll
      for (int c = 0; c < HD / 32; ++c) {
        uint32_t r[32];
        tmem_ld_32x32(lane_addr + c * 32, r);
        tmem_ld_wait();
        if (c == HD / 32 - 1) {
          tc_fence_before();
          mbar_arrive(bar(B_::DQ_READ));
        }
        if (lane == 0) tma_store_wait_read<1>();       // the piece before the last one has left its buffer
        __syncwarp();
        const uint32_t buf = stage + (c & 1) * 4096 + lane * 128;
#pragma unroll
        for (int j = 0; j < 8; ++j)
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(buf + ((j ^ (lane & 7)) << 4)), "r"(r[4 * j]),
                       "r"(r[4 * j + 1]), "r"(r[4 * j + 2]), "r"(r[4 * j + 3]) : "memory");
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          tma_reduce_add_3d(&p.tmdQ, stage + (c & 1) * 4096, h * HD + c * 32, i * BQ + (warp & 3) * 32, b);
          tma_store_commit();
        }
      }
    }
    if (lane == 0) tma_store_wait_all<0>();
  } else {
    // -------------------------------------------------------------------- P^T and dS^T: thread = key row, half of the queries
    const int row = threadIdx.x & 127;                 // == TMEM lane
    const int half = threadIdx.x >> 7;
    const uint32_t lane_addr = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    const int kj = k0 + row;
    const int kpos = p.k_off + kj * p.k_stride;
    // visible queries of this key: indices [q_first, q_end)
    int q_first = 0, q_end = 0x7fffffff;
    if (p.causal) q_first = kpos - p.q_off <= 0 ? 0 : (kpos - p.q_off + p.q_stride - 1) / p.q_stride;
    if (p.window > 0) {                                // q_pos <= kpos + window - 1
      const int last = kpos + p.window - 1 - p.q_off;
      q_end = last < 0 ? 0 : last / p.q_stride + 1;
    }
    if (kj >= p.Tk) q_end = 0;
    bool ok = true;
    for (int it = 0; it < n_iter; ++it) {
      const int i = i_lo + it % n_q;
      const float4* nl = reinterpret_cast<const float4*>(rows_s + (it & 1) * 256 + half * 64);
      const float4* nd = nl + 32;
      // does a mask or the end of the keys cut into this (query block, key block) pair?
      const int qpos_lo = p.q_off + i * BQ * p.q_stride, qpos_hi = p.q_off + (i * BQ + BQ - 1) * p.q_stride;
      const bool masked = (k0 + BKV > p.Tk) || (p.causal && kpos_hi > qpos_lo) ||
                          (p.window > 0 && kpos_lo <= qpos_hi - p.window);
      ok = mbar_wait(bar(B_::DO_FULL), it & 1, abort_smem, p.status, SITE_SMEM_FULL);   // L and Delta
      if (ok) ok = mbar_wait(bar(B_::S_FULL), it & 1, abort_smem, p.status, SITE_TMEM_FULL);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      float pv[64];
      const int first = q_first - i * BQ - half * 64, end = q_end - i * BQ - half * 64;
#pragma unroll
      for (int c = 0; c < 2; ++c) {                    // P of 32 queries takes 16 columns that have been read
        uint32_t rs[32], w[16];
        tmem_ld_32x32(lane_addr + C_S + half * 64 + c * 32, rs);
        tmem_ld_wait();
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const float4 L4 = nl[c * 8 + e];
          const float L[4] = {L4.x, L4.y, L4.z, L4.w};
#pragma unroll
          for (int u = 0; u < 4; ++u)
            pv[c * 32 + e * 4 + u] = ex2_approx(fmaf(__uint_as_float(rs[e * 4 + u]), p.scale_log2, L[u]));
        }
        if (masked) {
#pragma unroll
          for (int e = c * 32; e < c * 32 + 32; ++e)
            if (e < first || e >= end) pv[e] = 0.f;
        }
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          __nv_bfloat162 hb = __floats2bfloat162_rn(pv[c * 32 + 2 * e], pv[c * 32 + 2 * e + 1]);
          w[e] = *reinterpret_cast<uint32_t*>(&hb);
        }
        tmem_st_32x16(lane_addr + C_S + half * 64 + c * 16, w);
      }
      tmem_st_wait();
      tc_fence_before();
      mbar_arrive(bar(B_::P_FULL));
      ok = mbar_wait(bar(B_::DP_FULL), it & 1, abort_smem, p.status, SITE_TMEM_FULL);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t rp[32], w[16];
        tmem_ld_32x32(lane_addr + C_DP + half * 64 + c * 32, rp);
        tmem_ld_wait();
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const float4 d4 = nd[c * 8 + e];
          const int o = 4 * e;
          __nv_bfloat162 a = __floats2bfloat162_rn(pv[c * 32 + o] * fmaf(__uint_as_float(rp[o]), p.scale, d4.x),
                                                   pv[c * 32 + o + 1] * fmaf(__uint_as_float(rp[o + 1]), p.scale, d4.y));
          __nv_bfloat162 bb = __floats2bfloat162_rn(pv[c * 32 + o + 2] * fmaf(__uint_as_float(rp[o + 2]), p.scale, d4.z),
                                                    pv[c * 32 + o + 3] * fmaf(__uint_as_float(rp[o + 3]), p.scale, d4.w));
          w[2 * e] = *reinterpret_cast<uint32_t*>(&a);
          w[2 * e + 1] = *reinterpret_cast<uint32_t*>(&bb);
        }
        store_row32(sdS, row, half * 2 + c, w);
      }
      fence_proxy_async_smem();
      tc_fence_before();
      mbar_arrive(bar(B_::DS_FULL));
    }
    // ---- dK, dV of this key block (thread = key row, half of the head dimension)
    if (ok && n_iter > 0) {
      ok = mbar_wait(bar(B_::ACC_DONE), 0, abort_smem, p.status, SITE_TMEM_FULL);
      tc_fence_after();
    }
    ok = __all_sync(0xffffffffu, ok);
    if (ok && n_iter > 0) write_dkv<HD>(p, lane_addr + C_DV, lane_addr + C_DK, b, hk, kj, half);
    else if (n_iter == 0 && !p.dk_acc && half == 0) zero_dkv<HD>(p, b, hk, kj);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 13) {
    tc_fence_after();
    tmem_dealloc<1>(tmem, 512);
  }
}

// Delta = rowsum(dO o O) of the [rows, H, HD] matrices, stored as [B, H, T]; `zero` (fp32 [rows, H, HD], may be null) is
// cleared on the way: the accumulator of dQ.  HD / 8 lanes share a row of a head.
template <int HD>
__global__ void __launch_bounds__(256) delta_kernel(const __nv_bfloat16* __restrict__ dout, long long ld_do,
                                                    const __nv_bfloat16* __restrict__ out, long long ld_o, float* __restrict__ delta,
                                                    float* __restrict__ zero, int B, int T, int H) {
  constexpr int L = HD / 8;
  const long long total = (long long)B * T * H * L;
  // the turns are the warp's, so that all lanes meet at the shuffles; a row's lanes are in or out together (total % L == 0)
  for (long long first = blockIdx.x * 256ll + (threadIdx.x & ~31); first < total; first += gridDim.x * 256ll) {
    const long long idx = first + (threadIdx.x & 31);
    const bool in = idx < total;
    const int v = (int)(idx % L);
    const long long rh = idx / L;
    const int h = (int)(rh % H);
    const long long row = rh / H;
    float s = 0.f;
    if (in) {
      const uint4 a = __ldg(reinterpret_cast<const uint4*>(dout + row * ld_do + (long long)h * HD) + v);
      const uint4 o = __ldg(reinterpret_cast<const uint4*>(out + row * ld_o + (long long)h * HD) + v);
      const __nv_bfloat162* a2 = reinterpret_cast<const __nv_bfloat162*>(&a);
      const __nv_bfloat162* o2 = reinterpret_cast<const __nv_bfloat162*>(&o);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 x = __bfloat1622float2(a2[i]), y = __bfloat1622float2(o2[i]);
        s += x.x * y.x + x.y * y.y;
      }
    }
#pragma unroll
    for (int m = L / 2; m > 0; m >>= 1) s += __shfl_xor_sync(0xffffffffu, s, m);
    if (in && v == 0) {
      const long long b = row / T, t = row % T;
      delta[(b * H + h) * T + t] = s;
    }
    if (in && zero) {
      float4* z = reinterpret_cast<float4*>(zero + rh * HD) + 2 * v;
      z[0] = z[1] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
}

// [sample][row][column]: what a tile reads past the last row of its sample is zero, not the next sample's
static bool map3d(CUtensorMap* tm, const void* base, uint64_t cols, uint64_t rows, uint64_t samples, uint64_t ld) {
  cuuint64_t dims[3] = {cols, rows, samples};
  cuuint64_t strides[2] = {ld * 2, rows * ld * 2};
  cuuint32_t box[3] = {64, 128, 1};
  cuuint32_t es[3] = {1, 1, 1};
  return encode_tiled(tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, base, dims, strides, box, es, CU_TENSOR_MAP_SWIZZLE_128B);
}

static bool map_dq(CUtensorMap* tm, const float* dq, const MeshFlashArgs& f, long long ld, int hd) {
  cuuint64_t dims[3] = {(cuuint64_t)f.H * hd, (cuuint64_t)f.Tq, (cuuint64_t)f.B};
  cuuint64_t strides[2] = {(cuuint64_t)ld * 4, (cuuint64_t)f.Tq * ld * 4};
  cuuint32_t box[3] = {32, 32, 1};
  cuuint32_t es[3] = {1, 1, 1};
  return encode_tiled(tm, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, dq, dims, strides, box, es, CU_TENSOR_MAP_SWIZZLE_128B);
}

template <int HD>
static int launch(const MeshFlashBwdArgs* a, cudaStream_t stream) {
  constexpr int SMEM = 4 * 128 * HD * 2 + 2 * 128 * 128 * 2 + 1024 + 256;
  Params p;
  memset(&p, 0, sizeof(p));
  const MeshFlashArgs& f = a->fwd;
  if (!map3d(&p.tmQ, f.q, (uint64_t)f.q_cols, (uint64_t)f.Tq, (uint64_t)f.B, (uint64_t)f.ldq)) return last_error_code();
  if (!map3d(&p.tmK, f.k, (uint64_t)f.k_cols, (uint64_t)f.Tk, (uint64_t)f.B, (uint64_t)f.ldk)) return last_error_code();
  if (!map3d(&p.tmV, f.v, (uint64_t)f.v_cols, (uint64_t)f.Tk, (uint64_t)f.B, (uint64_t)f.ldv)) return last_error_code();
  if (!map3d(&p.tmdO, a->dout, (uint64_t)a->do_cols, (uint64_t)f.Tq, (uint64_t)f.B, (uint64_t)a->ld_do)) return last_error_code();
  if (!map_dq(&p.tmdQ, a->dq, f, a->ld_dq, HD)) return last_error_code();
  p.lse = f.lse; p.delta = a->delta; p.dq = a->dq; p.dk = (__nv_bfloat16*)a->dk; p.dv = (__nv_bfloat16*)a->dv;
  p.dk_acc = a->dk_acc; p.dv_acc = a->dv_acc;
  p.ld_dq = a->ld_dq; p.ld_dkv = a->ld_dkv;
  p.B = f.B; p.H = f.H; p.Hkv = f.Hkv; p.Tq = f.Tq; p.Tk = f.Tk;
  p.q_col0 = f.q_col0; p.k_col0 = f.k_col0; p.v_col0 = f.v_col0; p.do_col0 = a->do_col0;
  p.causal = f.causal; p.window = f.window;
  p.q_off = f.q_off; p.q_stride = f.q_stride > 0 ? f.q_stride : 1; p.k_off = f.k_off; p.k_stride = f.k_stride > 0 ? f.k_stride : 1;
  p.scale = f.scale; p.scale_log2 = f.scale * 1.4426950408889634f;
  p.status = (Status*)f.status;
  p.drop.p = f.dropout_p > 0.f ? f.dropout_p : 0.f;
  p.drop.inv_keep = p.drop.p > 0.f ? 1.f / (1.f - p.drop.p) : 1.f;
  p.drop.k0 = (uint32_t)(f.seed & 0xffffffffull) ^ (f.execution * 0x9E3779B9u);
  p.drop.k1 = (uint32_t)(f.seed >> 32);
  p.drop.site = f.site;
  p.head_off = f.head_off; p.heads_total = f.heads_total > 0 ? f.heads_total : f.H;
  if (p.drop.p > 0.f) {
    static bool configured = false;
    if (!configured) {
      MESH_CUDA_OK(cudaFuncSetAttribute(flash_bwd_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM));
      configured = true;
    }
    dim3 grid((f.Tk + BKV - 1) / BKV, f.Hkv, f.B);
    flash_bwd_kernel<HD><<<grid, THREADS, SMEM, stream>>>(p);
  } else {
    static bool configured = false;
    if (!configured) {
      MESH_CUDA_OK(cudaFuncSetAttribute(flash_bwd2_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg2<HD>::SMEM));
      configured = true;
    }
    dim3 grid(f.Hkv * f.B, (f.Tk + BKV - 1) / BKV);
    flash_bwd2_kernel<HD><<<grid, THREADS2, Cfg2<HD>::SMEM, stream>>>(p);
  }
  MESH_CUDA_OK(cudaGetLastError());
  return 0;
}

}  // namespace fab
}  // namespace mesh

extern "C" int mesh_flash_attention_bwd(const MeshFlashBwdArgs* a, void* stream) {
  using namespace mesh;
  const MeshFlashArgs& f = a->fwd;
  if (f.H % f.Hkv) return set_error(-2, "flash_attention_bwd: query heads must be a multiple of KV heads");
  if (f.lse == nullptr || a->delta == nullptr || a->dq == nullptr) return set_error(-2, "flash_attention_bwd: lse, delta and dq are required");
  if (a->ld_dq % 4 || a->ld_dkv % 8) return set_error(-2, "flash_attention_bwd: gradient leading dimensions are misaligned");
  switch (f.head_dim) {
    case 64: return fab::launch<64>(a, (cudaStream_t)stream);
    case 128: return fab::launch<128>(a, (cudaStream_t)stream);
    default: return set_error(-2, "flash_attention_bwd: head_dim must be 64 or 128 (dK and dV live in tensor memory)");
  }
}

extern "C" int mesh_attention_delta(const void* dout, long long ld_do, const void* out, long long ld_o, float* delta, float* zero,
                                    int B, int T, int H, int head_dim, void* stream) {
  using namespace mesh;
  if (ld_do % 8 || ld_o % 8 || (uintptr_t)dout % 16 || (uintptr_t)out % 16 || (uintptr_t)zero % 16)
    return set_error(-2, "attention_delta: rows must be 16-byte aligned");
  const long long groups = (long long)B * T * H * (head_dim / 8);
  if (groups <= 0) return 0;
  const unsigned grid = (unsigned)((groups + 255) / 256 < 148 * 16 ? (groups + 255) / 256 : 148 * 16);
#define MESH_DELTA(HD)                                                                                                       \
  fab::delta_kernel<HD><<<grid, 256, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)dout, ld_do, (const __nv_bfloat16*)out, \
                                                                ld_o, delta, zero, B, T, H)
  switch (head_dim) {
    case 64: MESH_DELTA(64); break;
    case 128: MESH_DELTA(128); break;
    case 256: MESH_DELTA(256); break;
    default: return set_error(-2, "attention_delta: head_dim must be 64, 128 or 256");
  }
#undef MESH_DELTA
  MESH_CUDA_OK(cudaGetLastError());
  return 0;
}
