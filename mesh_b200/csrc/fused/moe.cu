// Expert-parallel routed MoE: dispatch and combine fused with their all-to-all over NVLink peer memory,
// and the device-side planning that lets the expert GEMMs run as descriptor-driven tcgen05 launches
// with no host round trip.
//
//   moe_count     per-expert slot of every (token, choice) and this rank's expert histogram, pushed to
//                 every rank as 8-byte {count, sequence} words
//   moe_plan      from the P x E histogram matrix: where each sender's rows start inside each receiver's
//                 compact per-expert regions (padded to 256 rows), this rank's row layout, and the tile
//                 descriptor tables of its six grouped GEMMs (forward GLU / down, backward dgrad x2, wgrad x2)
//   moe_zero_pad  zero the padding rows of this rank's receive buffer (they feed the ragged-K wgrads)
//   moe_dispatch  every (token, choice) row is stored straight into the destination rank's expert region
//                 (optionally scaled: the backward pass sends w * dOut), then arrival counters are raised
//   moe_combine   after a ready exchange, every token pulls its k expert rows from the peers and sums them
//                 with its routing weights (optionally also the dot products <y, dOut> = gradients of the weights)
//
// Semantics follow the reference's GShard-style example (examples/ep.py:15-70): softmax router, top-k, slots
// assigned in token order, capacity-limited (rows past the receive capacity are dropped and their weight is
// zero), expert SwiGLU, weighted combine; its all-to-all is MPI_Alltoallv with per-pair counts
// (rdma/mesh_compile.py:1571-1579): counts are exchanged, blocks travel at their own sizes, never padded to the largest.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math_constants.h>
#include "moe_api.h"
#include "../device/check.cuh"
#include "../device/ptx.cuh"
#include "../gemm/gemm_api.h"
#include "../runtime/host_common.h"

namespace mesh {
namespace moe {

constexpr int R = MESH_MOE_MAX_RANKS;
constexpr int MAX_E = MESH_MOE_MAX_EXPERTS;

__device__ __forceinline__ void ll_store(uint2* p, uint32_t v, uint32_t seq) {
  asm volatile("st.volatile.global.v2.u32 [%0], {%1, %2};" ::"l"(p), "r"(v), "r"(seq) : "memory");
}
__device__ __forceinline__ bool ll_load(const uint2* p, uint32_t seq, uint32_t& v, Status* st) {
  uint2 w;
  unsigned long long t0 = 0;
  uint32_t it = 0;
  while (true) {
    asm volatile("ld.volatile.global.v2.u32 {%0, %1}, [%2];" : "=r"(w.x), "=r"(w.y) : "l"(p) : "memory");
    if (w.y == seq) { v = w.x; return true; }
    if (((++it) & 0x3ffu) == 0) {
      if (t0 == 0) t0 = globaltimer_ns();
      else if (globaltimer_ns() - t0 > MESH_WAIT_LIMIT_NS || status_aborted(st)) {
        status_record(st, MESH_TIMEOUT, SITE_PEER_FLAG, seq, w.y, (unsigned long long)p);
        return false;
      }
    }
  }
}

// ------------------------------------------------------------------------------------------- count
// slot[i] = number of earlier entries (token order) routed to the same expert.  A block ranks a chunk of 1024 entries
// (lanes that chose the same expert find each other with a match, warps are ordered through a small table in shared
// memory) and leaves the chunk's histogram in `work`; the block that finishes last turns the histograms into each
// chunk's starting slot per expert, adds them to the slots, and pushes the totals to every rank.
constexpr int COUNT_CHUNK = 1024;

__global__ void __launch_bounds__(COUNT_CHUNK)
moe_count_kernel(const int* __restrict__ idx, int n_entries, int* __restrict__ slot, int experts, int rank, int world,
                 int* __restrict__ work, uint2* c0, uint2* c1, uint2* c2, uint2* c3, uint2* c4, uint2* c5, uint2* c6,
                 uint2* c7, uint32_t seq) {
  __shared__ int cnt[32][MAX_E];            // [warp][expert]: entries of the warp, then entries of the warps before it
  __shared__ int last_s;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int chunks = gridDim.x;
  int* hist = work;                         // [chunks][experts]
  int* done = work + (long long)chunks * experts;
  for (int j = threadIdx.x; j < 32 * MAX_E; j += blockDim.x) (&cnt[0][0])[j] = 0;
  __syncthreads();
  const int i = blockIdx.x * COUNT_CHUNK + threadIdx.x;
  const bool valid = i < n_entries;
  const int e = valid ? idx[i] : -1 - lane;                                  // invalid lanes match nobody
  const bool good = valid && e >= 0 && e < experts;
  const unsigned same = __match_any_sync(0xffffffffu, e);
  const int in_warp = __popc(same & ((1u << lane) - 1u));
  if (good && in_warp == 0) cnt[warp][e] = __popc(same);
  __syncthreads();
  if ((int)threadIdx.x < experts) {                                          // exclusive scan over the warps
    int run = 0;
    for (int w = 0; w < 32; ++w) {
      const int c = cnt[w][threadIdx.x];
      cnt[w][threadIdx.x] = run;
      run += c;
    }
    hist[(long long)blockIdx.x * experts + threadIdx.x] = run;
  }
  __syncthreads();
  if (good) slot[i] = cnt[warp][e] + in_warp;
  else if (valid) slot[i] = 0;
  // ---- the last block to finish completes the slots
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    const int d = atomicAdd(done, 1);
    last_s = (d == chunks - 1);
    if (last_s) *done = 0;                                                   // ready for the next launch
  }
  __syncthreads();
  if (!last_s) return;
  __threadfence();
  if ((int)threadIdx.x < experts) {
    int run = 0;
    int* h = hist + threadIdx.x;
    for (int c0 = 0; c0 < chunks; c0 += 8) {                                 // eight loads in flight, not one
      int n[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) n[u] = c0 + u < chunks ? __ldcg(h + (long long)(c0 + u) * experts) : 0;
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        if (c0 + u < chunks) h[(long long)(c0 + u) * experts] = run;
        run += n[u];
      }
    }
    if (world > 0) {
      uint2* peers[8] = {c0, c1, c2, c3, c4, c5, c6, c7};
      // count matrix on every rank: [parity][src rank][expert]
      for (int r = 0; r < world; ++r)
        ll_store(peers[r] + ((long long)(seq & 1u) * world + rank) * experts + threadIdx.x, (uint32_t)run, seq);
    }
  }
  __syncthreads();
  for (int j = COUNT_CHUNK + (int)threadIdx.x; j < n_entries; j += COUNT_CHUNK) {   // chunk 0 starts at slot 0
    const int ej = idx[j];
    if (ej >= 0 && ej < experts) slot[j] = __ldcg(slot + j) + hist[(long long)(j / COUNT_CHUNK) * experts + ej];
  }
}

// ------------------------------------------------------------------------------------------- plan
struct PlanArgs {
  const uint2* counts;         // this rank's count matrix [2][world][experts]
  uint32_t seq;
  int rank, world, experts, cap_rows;
  int d_model, d_ff;           // expert shapes: W1 [2*d_ff, d_model], W2 [d_model, d_ff]
  int* send_base;              // [experts]: first row for this sender in the destination's region of expert e
  int* layout;                 // [3 * local experts + 2]: n_e..., base_e..., padded_e..., total_rows, dropped flag
  MeshTileDesc* t_glu; MeshTileDesc* t_down; MeshTileDesc* t_dh; MeshTileDesc* t_dx; MeshTileDesc* t_dw2; MeshTileDesc* t_dw1;
  int* n_tiles;                // [8]: lengths of the six tables, then two counters that the launch leaves at zero
  int max_tiles;
  Status* status;
};

// Every CTA works out the same layout (a few microseconds of a 60 us kernel when one CTA wrote all tables, some fifteen
// thousand 32-byte records at 64 experts); the first one stores it, and the experts' records are shared out.  Each waits for
// the counts by itself, so one may give up where another did not: the last to finish publishes the tables' lengths, and
// publishes zeros when any of them wrote no records.
constexpr int PLAN_CTAS = 16;

__global__ void __launch_bounds__(512) moe_plan_kernel(const PlanArgs a) {
  __shared__ int C[R][MAX_E];
  __shared__ int n_loc[MAX_E], base_loc[MAX_E], pad_loc[MAX_E];
  __shared__ int ok_s;
  const int E = a.experts, P = a.world, El = E / P;
  if (threadIdx.x == 0) ok_s = 1;
  __syncthreads();
  for (int i = threadIdx.x; i < P * E; i += blockDim.x) {
    uint32_t v = 0;
    if (!ll_load(a.counts + (long long)(a.seq & 1u) * P * E + i, a.seq, v, a.status)) ok_s = 0;
    C[i / E][i % E] = (int)v;
  }
  __syncthreads();
  const bool first = blockIdx.x == 0;
  __shared__ int off[6][MAX_E + 1];
  __shared__ int last_s, failed_s;
  auto publish = [&](bool ok) {            // all threads of the CTA
    __threadfence();                       // this thread's records before this CTA's mark
    __syncthreads();
    if (threadIdx.x == 0) {
      if (!ok) atomicAdd(a.n_tiles + 7, 1);
      __threadfence();
      last_s = atomicAdd(a.n_tiles + 6, 1) == (int)gridDim.x - 1;
      if (last_s) {
        failed_s = atomicExch(a.n_tiles + 7, 0);
        a.n_tiles[6] = 0;                  // ready for the next launch
      }
    }
    __syncthreads();
    if (last_s && threadIdx.x < 6) a.n_tiles[threadIdx.x] = failed_s == 0 ? min(off[threadIdx.x][El], a.max_tiles) : 0;
  };
  if (!ok_s) {
    publish(false);
    return;
  }
  // every destination's layout is the same function of the matrix; this rank needs all of them as a sender
  if (threadIdx.x < E) {
    const int e = threadIdx.x, d = e / El, el = e % El;
    int base = 0;
    for (int k = 0; k < el; ++k) {
      int n = 0;
      for (int s = 0; s < P; ++s) n += C[s][d * El + k];
      base += (n + 255) / 256 * 256;
    }
    int before = 0;
    for (int s = 0; s < a.rank; ++s) before += C[s][e];
    if (first) a.send_base[e] = base + before;
    if (d == a.rank) {
      int n = 0;
      for (int s = 0; s < P; ++s) n += C[s][e];
      n_loc[el] = n;
      base_loc[el] = base;
      pad_loc[el] = (n + 255) / 256 * 256;
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int total = 0, dropped = 0;
    for (int el = 0; el < El; ++el) {
      // rows past the capacity are dropped by the senders; the receiver clips its regions the same way
      if (base_loc[el] + pad_loc[el] > a.cap_rows) {
        dropped = 1;
        const int room = max(0, a.cap_rows - base_loc[el]) / 256 * 256;
        pad_loc[el] = min(pad_loc[el], room);
        n_loc[el] = min(n_loc[el], pad_loc[el]);
      }
      total = max(total, base_loc[el] + pad_loc[el]);
    }
    if (first) {
      a.layout[3 * El] = total;
      a.layout[3 * El + 1] = dropped;
    }
  }
  __syncthreads();
  if (first && (int)threadIdx.x < El) {
    a.layout[threadIdx.x] = n_loc[threadIdx.x];
    a.layout[El + threadIdx.x] = base_loc[threadIdx.x];
    a.layout[2 * El + threadIdx.x] = pad_loc[threadIdx.x];
  }
  // ---- tile tables (pair tiles: 256 output rows each).  Table t of expert el holds cnt[t][el] descriptors starting at
  // off[t][el]; thread 0 lays the offsets out (6 x local experts additions), then every warp writes the descriptors of
  // its experts, a lane per tile: the tables are thousands of 32-byte records, far too many for one thread.
  const int D = a.d_model, F = a.d_ff;
  const int ntn[6] = {(F + 127) / 128, (D + 255) / 256, (F + 255) / 256, (D + 255) / 256, (F + 255) / 256, (D + 255) / 256};
  const int dw_mt[2] = {(D + 255) / 256, (2 * F + 255) / 256};
  if (threadIdx.x < 6) {
    const int t = threadIdx.x;
    int n = 0;
    for (int el = 0; el < El; ++el) {
      off[t][el] = n;
      const int rows = pad_loc[el];
      n += t < 4 ? (rows / 256) * ntn[t] : (rows >= 64 ? dw_mt[t - 4] * ntn[t] : 0);
    }
    off[t][El] = n;
  }
  __syncthreads();
  MeshTileDesc* const tab[6] = {a.t_glu, a.t_down, a.t_dh, a.t_dx, a.t_dw2, a.t_dw1};
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
  for (int el = blockIdx.x + gridDim.x * warp; el < El; el += gridDim.x * nwarps) {
    const int base = base_loc[el], kb = pad_loc[el] / 64;
#pragma unroll
    for (int t = 0; t < 6; ++t) {
      const int cnt = off[t][el + 1] - off[t][el];
      for (int j = lane; j < cnt; j += 32) {
        const int at = off[t][el] + j;
        if (at >= a.max_tiles) break;
        const int mt = j / ntn[t], nt = j - mt * ntn[t];
        const int row = base + mt * 256;
        MeshTileDesc d;
        if (t == 0) d = MeshTileDesc{row, 0, D / 64, el * 2 * F + nt * 128, 0, row, nt * 128, 0};            // h = act(x W1g^T) * (x W1u^T)
        else if (t == 1) d = MeshTileDesc{row, 0, F / 64, el * D + nt * 256, 0, row, nt * 256, 0};           // y = h W2^T
        else if (t == 2) d = MeshTileDesc{row, 0, D / 64, nt * 256, el * D, row, nt * 256, 0};               // dH = dY W2   (W2 stacked [El*D, F], MN-major)
        else if (t == 3) d = MeshTileDesc{row, 0, (2 * F) / 64, nt * 256, el * 2 * F, row, nt * 256, 0};     // dX = dGU W1  (W1 stacked [El*2F, D], MN-major)
        else if (t == 4) d = MeshTileDesc{mt * 256, base, kb, nt * 256, 0, el * D + mt * 256, nt * 256, D - mt * 256};  // dW2[el] = dY^T h   [D, F]
        else d = MeshTileDesc{mt * 256, base, kb, nt * 256, 0, el * 2 * F + mt * 256, nt * 256, 2 * F - mt * 256};          // dW1[el] = dGU^T x  [2F, D]
        tab[t][at] = d;
      }
    }
  }
  publish(true);
}

// ------------------------------------------------------------------------------------------- zero padding rows
__global__ void moe_zero_pad_kernel(__nv_bfloat16* __restrict__ buf, const int* __restrict__ layout, int local_experts,
                                    int d_model) {
  const int el = blockIdx.y;
  const int n = layout[el], base = layout[local_experts + el], pad = layout[2 * local_experts + el];
  const long long vec_per_row = d_model / 8;
  const long long total = (long long)(pad - n) * vec_per_row;
  uint4* p = reinterpret_cast<uint4*>(buf + (long long)(base + n) * d_model);
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x)
    p[i] = make_uint4(0, 0, 0, 0);
}

// ------------------------------------------------------------------------------------------- dispatch
struct DispatchArgs {
  const __nv_bfloat16* x; int tokens, k, d_model;
  const int* idx; const int* slot; const int* send_base; const float* scale;     // scale [tokens, k] or nullptr
  int* meta;                                   // [tokens, k]: row in the destination buffer, or -1 when dropped
  int local_experts, cap_rows, rank, world;
  __nv_bfloat16* recv[R];                      // every rank's receive buffer [cap_rows, d_model]
  uint32_t* arrived[R];                        // every rank's arrival counter for this buffer
  Status* status;
};

__global__ void __launch_bounds__(256) moe_dispatch_kernel(const DispatchArgs a) {
  const int warps = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int vec = a.d_model / 8;
  // A warp owns a token: its row is read once and stored to the k rows that were assigned to it (a warp per stored row
  // read it k times): 8192 tokens of 2048, six choices, 49 us now, 61 before.
  for (int t = blockIdx.x * warps + warp; t < a.tokens; t += gridDim.x * warps) {
    const uint4* src = reinterpret_cast<const uint4*>(a.x + (long long)t * a.d_model);
    for (int j0 = 0; j0 < a.k; j0 += 32) {
      // lane j: where choice j0 + j of this token goes
      unsigned long long dst = 0;
      float s = 1.f;
      const int i = t * a.k + j0 + lane;
      if (j0 + lane < a.k) {
        const int e = a.idx[i];
        if (MESH_CHECK_INDEX(e, a.local_experts * a.world, a.status)) {           // an expert id from the router
          const int row = a.send_base[e] + a.slot[i];
          if (MESH_CHECK_INDEX(row, 1ll << 30, a.status)) {                       // negative: a broken plan
            const bool fits = row < a.cap_rows;
            a.meta[i] = fits ? row : -1;
            if (fits) dst = reinterpret_cast<unsigned long long>(a.recv[e / a.local_experts] + (long long)row * a.d_model);
          }
        }
        if (a.scale) s = a.scale[i];
      }
      const int n = min(32, a.k - j0);
      for (int base = 0; base < vec; base += 4 * 32) {
        const int v0 = base + lane;
        uint4 q[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (v0 + u * 32 < vec) q[u] = __ldg(src + v0 + u * 32);
        for (int j = 0; j < n; ++j) {
          uint4* d = reinterpret_cast<uint4*>(__shfl_sync(0xffffffffu, dst, j));
          const float sj = __shfl_sync(0xffffffffu, s, j);
          if (d == nullptr) continue;                                             // the same for the whole warp
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            if (v0 + u * 32 >= vec) break;
            uint4 o = q[u];
            if (a.scale) {
              __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
              for (int c = 0; c < 4; ++c) {
                const float2 f = __bfloat1622float2(h[c]);
                h[c] = __floats2bfloat162_rn(f.x * sj, f.y * sj);
              }
            }
            d[v0 + u * 32] = o;
          }
        }
      }
    }
  }
  __syncthreads();                      // the signalling threads' system-scope release covers the block's stores
  if ((int)threadIdx.x < a.world) red_release_sys_add(a.arrived[threadIdx.x], 1u);
}

// ------------------------------------------------------------------------------------------- ready exchange
__global__ void moe_signal_kernel(int world, uint32_t* r0, uint32_t* r1, uint32_t* r2, uint32_t* r3, uint32_t* r4,
                                  uint32_t* r5, uint32_t* r6, uint32_t* r7) {
  uint32_t* peers[8] = {r0, r1, r2, r3, r4, r5, r6, r7};
  __threadfence_system();
  if ((int)threadIdx.x < world) red_release_sys_add(peers[threadIdx.x], 1u);
}

// ------------------------------------------------------------------------------------------- combine
struct CombineArgs {
  int tokens, k, d_model, local_experts, world;
  const int* idx; const int* meta; const float* weight;        // weight nullptr: plain sum (backward of dispatch)
  const __nv_bfloat16* src[R];                 // every rank's expert-output buffer [cap_rows, d_model]
  int cap_rows;                                // rows of every expert-output buffer (checked build)
  const uint32_t* ready; uint32_t ready_expect;               // this rank's counter: all peers finished their experts
  __nv_bfloat16* out;                          // [tokens, d_model]
  const __nv_bfloat16* dot_with; float* dots;  // optional: dots[t, j] = <row, dot_with[t]>
  const __nv_bfloat16* addend;                 // optional [tokens, d_model]: added to the sum before it is rounded
  Status* status;
};

// J rows of a token are read together (one after the other, each behind its index loads, the pass ran at 3 TB/s).  J and the
// kind of result are template parameters because the rows in flight live in registers: 8192 tokens of 2048 with six rows
// each take 55 us (sum) and 52 us (dots), 73 and 99 before.
template <int J, bool DOTS>
__global__ void __launch_bounds__(256, 3) moe_combine_kernel(const CombineArgs a) {
  __shared__ int ok_s;
  if (threadIdx.x == 0) ok_s = wait_flag_ge(a.ready, a.ready_expect, a.status, SITE_PEER_FLAG) ? 1 : 0;
  __syncthreads();
  if (!ok_s) return;
  const int warps = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int vec = a.d_model / 8;       // 16-byte vectors per row; a lane owns vectors lane, lane+32, ...
  for (int t = blockIdx.x * warps + warp; t < a.tokens; t += gridDim.x * warps) {
    // lane j: the row of choice j (k <= 32), null when it was dropped
    unsigned long long mine = 0;
    float mw = 1.f;
    if (lane < a.k) {
      const int i = t * a.k + lane, row = a.meta[i];
      if (row >= 0) {
        const int dest = a.idx[i] / a.local_experts;
        if (MESH_CHECK_INDEX(dest, a.world, a.status) && MESH_CHECK_INDEX(row, a.cap_rows, a.status))
          mine = reinterpret_cast<unsigned long long>(a.src[dest] + (long long)row * a.d_model);
      }
      if (a.weight) mw = a.weight[i];
    }
    const uint4* src[J];
    float w[J];
    auto pick = [&](int j0) {
#pragma unroll
      for (int j = 0; j < J; ++j) {
        const unsigned long long p = __shfl_sync(0xffffffffu, mine, (j0 + j) & 31);
        w[j] = __shfl_sync(0xffffffffu, mw, (j0 + j) & 31);
        src[j] = j0 + j < a.k ? reinterpret_cast<const uint4*>(p) : nullptr;
      }
    };
    pick(0);
    if constexpr (!DOTS) {
      for (int base = 0; base < vec; base += 32) {
        const int v = base + lane;
        const bool in = v < vec;
        float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        uint4 extra = make_uint4(0, 0, 0, 0);
        if (a.addend && in) extra = __ldg(reinterpret_cast<const uint4*>(a.addend + (long long)t * a.d_model) + v);
        for (int j0 = 0; j0 < a.k; j0 += J) {
          if (a.k > J) pick(j0);
          uint4 q[J];
#pragma unroll
          for (int j = 0; j < J; ++j)
            if (src[j] != nullptr && in) q[j] = __ldcg(src[j] + v);
#pragma unroll
          for (int j = 0; j < J; ++j) {
            if (src[j] == nullptr || !in) continue;
            const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&q[j]);
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              const float2 f = __bfloat1622float2(h[c]);
              acc[2 * c] += w[j] * f.x;
              acc[2 * c + 1] += w[j] * f.y;
            }
          }
        }
        if (!in) continue;
        const __nv_bfloat162* e = reinterpret_cast<const __nv_bfloat162*>(&extra);
        uint4 o;
        __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const float2 f = __bfloat1622float2(e[c]);
          h[c] = __floats2bfloat162_rn(acc[2 * c] + f.x, acc[2 * c + 1] + f.y);
        }
        reinterpret_cast<uint4*>(a.out + (long long)t * a.d_model)[v] = o;
      }
    }
    if constexpr (DOTS) {
      for (int j0 = 0; j0 < a.k; j0 += J) {
        if (a.k > J) pick(j0);
        float dot[J];
#pragma unroll
        for (int j = 0; j < J; ++j) dot[j] = 0.f;
        for (int v = lane; v < vec; v += 32) {
          const uint4 g = __ldg(reinterpret_cast<const uint4*>(a.dot_with + (long long)t * a.d_model) + v);
          uint4 q[J];
#pragma unroll
          for (int j = 0; j < J; ++j) {
            q[j] = make_uint4(0, 0, 0, 0);
            if (src[j] != nullptr) q[j] = __ldcg(src[j] + v);
          }
          const __nv_bfloat162* gh = reinterpret_cast<const __nv_bfloat162*>(&g);
#pragma unroll
          for (int j = 0; j < J; ++j) {
            const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&q[j]);
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              const float2 f = __bfloat1622float2(h[c]), gg = __bfloat1622float2(gh[c]);
              dot[j] += f.x * gg.x + f.y * gg.y;
            }
          }
        }
#pragma unroll
        for (int j = 0; j < J; ++j) {
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) dot[j] += __shfl_xor_sync(0xffffffffu, dot[j], o);
          if (lane == j && j0 + j < a.k) a.dots[t * a.k + j0 + j] = src[j] != nullptr ? dot[j] : 0.f;
        }
      }
    }
  }
}

// Weight gradients of the experts that got no rows: their tables hold no tiles, so nothing else writes them.
__global__ void __launch_bounds__(256) moe_zero_unused_kernel(uint4* __restrict__ dw1, long long vec1, uint4* __restrict__ dw2,
                                                              long long vec2, const int* __restrict__ layout, int local_experts,
                                                              const int* __restrict__ n_tiles) {
  const int el = blockIdx.y;
  if (layout[2 * local_experts + el] >= 64 && n_tiles[4] > 0) return;
  for (long long i = blockIdx.x * 256ll + threadIdx.x; i < vec1; i += gridDim.x * 256ll) dw1[el * vec1 + i] = make_uint4(0, 0, 0, 0);
  for (long long i = blockIdx.x * 256ll + threadIdx.x; i < vec2; i += gridDim.x * 256ll) dw2[el * vec2 + i] = make_uint4(0, 0, 0, 0);
}

// Gradient of the routing weights w = top-k of softmax(logits + bias), renormalised over the k, through to the logits; a warp
// per token.  dots[t, j]: gradient of w_j (0 counts for a dropped choice).  With p the softmax and S the sum of the chosen
// p, d p_j = (g_j - sum_i w_i g_i) / S on the chosen experts and 0 elsewhere; sum_e p_e d p_e vanishes, so the softmax's
// backward is d logits = p d p.
__global__ void __launch_bounds__(256) moe_router_bwd_kernel(const __nv_bfloat16* __restrict__ logits, const float* __restrict__ bias,
                                                             const int* __restrict__ idx, const int* __restrict__ meta,
                                                             const float* __restrict__ dots, __nv_bfloat16* __restrict__ dlogits,
                                                             int tokens, int experts, int k) {
  constexpr int PER = MAX_E / 32;
  const int warps = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int t = blockIdx.x * warps + warp; t < tokens; t += gridDim.x * warps) {
    float v[PER];
    float mx = -CUDART_INF_F;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int e = lane + 32 * i;
      v[i] = e < experts ? __bfloat162float(logits[(long long)t * experts + e]) + (bias ? bias[e] : 0.f) : -CUDART_INF_F;
      mx = fmaxf(mx, v[i]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    float sum = 0.f;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      v[i] = lane + 32 * i < experts ? expf(v[i] - mx) : 0.f;
      sum += v[i];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    // lane j: the j-th choice
    const int i = t * k + lane;
    const int e = lane < k ? idx[i] : 0;
    const float g = lane < k && meta[i] >= 0 ? dots[i] : 0.f;
    float pe = 0.f;
#pragma unroll
    for (int r = 0; r < PER; ++r) {
      const float got = __shfl_sync(0xffffffffu, v[r], e & 31);
      if ((e >> 5) == r) pe = got;
    }
    pe = lane < k ? pe / sum : 0.f;
    float S = pe, wg = pe * g;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      S += __shfl_xor_sync(0xffffffffu, S, o);
      wg += __shfl_xor_sync(0xffffffffu, wg, o);
    }
    const float d = pe * (g - wg / S) / S;
#pragma unroll
    for (int r = 0; r < PER; ++r) {
      const int at = lane + 32 * r;
      float out = 0.f;
      for (int j = 0; j < k; ++j) {
        const int ej = __shfl_sync(0xffffffffu, e, j);
        const float dj = __shfl_sync(0xffffffffu, d, j);
        if (ej == at) out = dj;
      }
      if (at < experts) dlogits[(long long)t * experts + at] = __float2bfloat16_rn(out);
    }
  }
}

}  // namespace moe
}  // namespace mesh

using namespace mesh;
using namespace mesh::moe;

extern "C" int mesh_moe_count_work_ints(int n_entries, int experts) {
  return (n_entries + COUNT_CHUNK - 1) / COUNT_CHUNK * experts + 1;
}

extern "C" int mesh_moe_count(const int* idx, int n_entries, int* slot, int experts, int rank, int world,
                              void* const* count_ptrs, uint32_t seq, int* work, void* stream) {
  if (experts > MAX_E || world > R || experts % world) return set_error(-2, "moe_count: experts <= %d, divisible by world <= %d", MAX_E, R);
  if (n_entries < 1 || work == nullptr) return set_error(-2, "moe_count: no entries or no work buffer");
  uint2* c[8] = {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr};
  for (int r = 0; r < world; ++r) c[r] = (uint2*)count_ptrs[r];
  const int chunks = (n_entries + COUNT_CHUNK - 1) / COUNT_CHUNK;
  moe_count_kernel<<<chunks, COUNT_CHUNK, 0, (cudaStream_t)stream>>>(idx, n_entries, slot, experts, rank, world, work, c[0],
                                                                     c[1], c[2], c[3], c[4], c[5], c[6], c[7], seq);
  MESH_CUDA_OK(cudaGetLastError());
  return 0;
}

extern "C" int mesh_moe_plan(const MeshMoePlan* m, void* stream) {
  if (m->d_model % 256 || m->d_ff % 64) return set_error(-2, "moe_plan: d_model %% 256 and d_ff %% 64 must be 0");
  PlanArgs a;
  a.counts = (const uint2*)m->counts; a.seq = m->seq; a.rank = m->rank; a.world = m->world; a.experts = m->experts;
  a.cap_rows = m->cap_rows; a.d_model = m->d_model; a.d_ff = m->d_ff;
  a.send_base = m->send_base; a.layout = m->layout;
  a.t_glu = (MeshTileDesc*)m->tables[0]; a.t_down = (MeshTileDesc*)m->tables[1]; a.t_dh = (MeshTileDesc*)m->tables[2];
  a.t_dx = (MeshTileDesc*)m->tables[3]; a.t_dw2 = (MeshTileDesc*)m->tables[4]; a.t_dw1 = (MeshTileDesc*)m->tables[5];
  a.n_tiles = m->n_tiles; a.max_tiles = m->max_tiles; a.status = (Status*)m->status;
  moe_plan_kernel<<<PLAN_CTAS, 512, 0, (cudaStream_t)stream>>>(a);
  MESH_CUDA_OK(cudaGetLastError());
  return 0;
}

extern "C" int mesh_moe_zero_pad(void* buf, const int* layout, int local_experts, int d_model, void* stream) {
  dim3 grid(32, local_experts);
  moe_zero_pad_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>((__nv_bfloat16*)buf, layout, local_experts, d_model);
  MESH_CUDA_OK(cudaGetLastError());
  return 0;
}

extern "C" int mesh_moe_dispatch(const MeshMoeDispatch* m, void* stream) {
  if (m->d_model % 8) return set_error(-2, "moe_dispatch: d_model must be a multiple of 8");
  DispatchArgs a;
  a.x = (const __nv_bfloat16*)m->x; a.tokens = m->tokens; a.k = m->k; a.d_model = m->d_model;
  a.idx = m->idx; a.slot = m->slot; a.send_base = m->send_base; a.scale = m->scale; a.meta = m->meta;
  a.local_experts = m->local_experts; a.cap_rows = m->cap_rows; a.rank = m->rank; a.world = m->world;
  for (int r = 0; r < m->world; ++r) { a.recv[r] = (__nv_bfloat16*)m->recv[r]; a.arrived[r] = (uint32_t*)m->arrived[r]; }
  a.status = (Status*)m->status;
  moe_dispatch_kernel<<<MESH_MOE_DISPATCH_BLOCKS, 256, 0, (cudaStream_t)stream>>>(a);
  MESH_CUDA_OK(cudaGetLastError());
  return 0;
}

extern "C" int mesh_moe_signal(int world, void* const* ready_ptrs, void* stream) {
  uint32_t* r[8] = {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr};
  for (int i = 0; i < world; ++i) r[i] = (uint32_t*)ready_ptrs[i];
  moe_signal_kernel<<<1, 32, 0, (cudaStream_t)stream>>>(world, r[0], r[1], r[2], r[3], r[4], r[5], r[6], r[7]);
  MESH_CUDA_OK(cudaGetLastError());
  return 0;
}

extern "C" int mesh_moe_combine(const MeshMoeCombine* m, void* stream) {
  if (m->k > 32) return set_error(-2, "moe_combine: at most 32 choices per token");
  CombineArgs a;
  a.tokens = m->tokens; a.k = m->k; a.d_model = m->d_model; a.local_experts = m->local_experts; a.world = m->world;
  a.idx = m->idx; a.meta = m->meta; a.weight = m->weight;
  for (int r = 0; r < m->world; ++r) a.src[r] = (const __nv_bfloat16*)m->src[r];
  a.ready = (const uint32_t*)m->ready; a.ready_expect = m->ready_expect;
  a.out = (__nv_bfloat16*)m->out; a.dot_with = (const __nv_bfloat16*)m->dot_with; a.dots = m->dots;
  a.status = (Status*)m->status;
  a.cap_rows = m->cap_rows > 0 ? m->cap_rows : (1 << 30);
  a.addend = (const __nv_bfloat16*)m->addend;
  int grid = (m->tokens + 7) / 8;
  if (grid > 148 * 8) grid = 148 * 8;
#define MESH_COMBINE(DOTS)                                                                          \
  do {                                                                                              \
    if (a.k <= 2) moe_combine_kernel<2, DOTS><<<grid, 256, 0, (cudaStream_t)stream>>>(a);           \
    else if (a.k <= 4) moe_combine_kernel<4, DOTS><<<grid, 256, 0, (cudaStream_t)stream>>>(a);      \
    else if (a.k <= 6) moe_combine_kernel<6, DOTS><<<grid, 256, 0, (cudaStream_t)stream>>>(a);      \
    else moe_combine_kernel<8, DOTS><<<grid, 256, 0, (cudaStream_t)stream>>>(a);                    \
  } while (0)
  if (a.out) MESH_COMBINE(false);
  if (a.dots) MESH_COMBINE(true);
#undef MESH_COMBINE
  MESH_CUDA_OK(cudaGetLastError());
  return 0;
}

extern "C" int mesh_moe_zero_unused(void* dw1, long long elems1, void* dw2, long long elems2, const int* layout, int local_experts,
                                    const int* n_tiles, void* stream) {
  if (elems1 % 8 || elems2 % 8) return set_error(-2, "moe_zero_unused: expert matrices must be multiples of 8 elements");
  dim3 grid(16, local_experts);
  moe_zero_unused_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>((uint4*)dw1, elems1 / 8, (uint4*)dw2, elems2 / 8, layout, local_experts,
                                                                n_tiles);
  MESH_CUDA_OK(cudaGetLastError());
  return 0;
}

extern "C" int mesh_moe_router_bwd(const void* logits, const float* bias, const int* idx, const int* meta, const float* dots,
                                   void* dlogits, int tokens, int experts, int k, void* stream) {
  if (experts > MAX_E || k < 1 || k > 32) return set_error(-2, "moe_router_bwd: experts <= %d, k <= 32", MAX_E);
  int grid = (tokens + 7) / 8;
  if (grid > 148 * 8) grid = 148 * 8;
  if (grid < 1) return 0;
  moe_router_bwd_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)logits, bias, idx, meta, dots,
                                                               (__nv_bfloat16*)dlogits, tokens, experts, k);
  MESH_CUDA_OK(cudaGetLastError());
  return 0;
}
