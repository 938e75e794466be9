// Split-KV attention for decoding: one query token per sequence, grouped-query heads, optional
// sliding window.  Grid = (splits, kv_heads, batch): a CTA scores its slice of the keys for all the
// query heads that share one KV head (so K and V are read once per group), keeps the online-softmax
// triple (m, l, acc) per head, and the last CTA of a (sequence, kv head) to finish merges the
// partials.  Semantics: blockwise attention with (m, s, acc) merging and GQA by viewing query heads
// as [kv_heads, group] (compiler/mesh_compiler/operations.py:7081-7166, :7072-7078); the window is
// the E2B-class local layer (design/e2b-crossover-2026-09-16.md:42-52).
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math_constants.h>
#include "decode_api.h"
#include "../runtime/host_common.h"
#include <cstring>

namespace mesh {
namespace decode_att {

constexpr int ATT_THREADS = 256;
constexpr int ATT_WARPS = 8;
constexpr int MAX_GROUPS = 8;    // query heads per KV head, at most
constexpr int MAX_HD = 256;

struct AttArgs {
  const __nv_bfloat16* q; const __nv_bfloat16* kc; const __nv_bfloat16* vc; const int* pos;
  __nv_bfloat16* out; float* scratch; int* counters;
  int q_heads, kv_heads, max_seq, window; float scale; int splits, T;
  int B, head_dim;                                   // used by callers that loop over the work items themselves
  int unaligned;                                     // q or a cache does not start on a multiple of a lane's bytes
};

struct AttBlockSync { __device__ __forceinline__ void operator()() const { __syncthreads(); } };

// PER consecutive bf16 of a cache row, as stored
template <int PER> struct Raw;
template <> struct Raw<8> { uint4 v; };
template <> struct Raw<4> { uint2 v; };
template <> struct Raw<2> { uint32_t v; };
template <int PER>
__device__ __forceinline__ void widen(const Raw<PER>& r, float (&f)[PER]) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&r);
#pragma unroll
  for (int i = 0; i < PER / 2; ++i) {
    const float2 t = __bfloat1622float2(h[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}

// ONE_BY_ONE: the address is not a multiple of the vector's size.
template <int PER, bool ONE_BY_ONE>
__device__ __forceinline__ Raw<PER> load_raw(const __nv_bfloat16* p) {
  Raw<PER> r;
  if (!ONE_BY_ONE) return *reinterpret_cast<const Raw<PER>*>(p);
  __nv_bfloat16* h = reinterpret_cast<__nv_bfloat16*>(&r);
#pragma unroll
  for (int i = 0; i < PER; ++i) h[i] = p[i];
  return r;
}
inline bool unaligned(const void* q, const void* kc, const void* vc, int head_dim) {
  return (((uintptr_t)q | (uintptr_t)kc | (uintptr_t)vc) % (uintptr_t)(head_dim / 32 * 2)) != 0;
}

// Running softmax of one warp over its keys.  A lane owns HD / 32 consecutive dims of K, V and the accumulators; m and l
// are those of head `lane / 2 % MAXG`, the head whose scores the lane holds after the reduction below.
template <int HD, int MAXG>
struct WarpState {
  static constexpr int PER = HD / 32;
  static constexpr int KEYS = 16 / MAXG;              // keys a warp takes at a time: 16 scores, two lanes each
  float m, l, acc[MAXG][PER];
};

// Keys of this warp: KEYS consecutive ones starting at lo + gw * KEYS, then every `warps` * KEYS further, up to hi.  All
// loads of a step are issued together (a key costs a trip to L2 or HBM, not two); the 16 partial dot products are
// reduced with 16 shuffles instead of 5 each, and every lane then works on one score: one exponential, not 16.
// ONE_BY_ONE: see load_raw; a template, since a branch at the loads keeps them from being issued together (23 us instead of 18).
template <int HD, int MAXG, bool ONE_BY_ONE>
__device__ __forceinline__ void scan_keys(const AttArgs& A, int kvh, int b, int lo, int hi, int gw, int warps,
                                          WarpState<HD, MAXG>& st) {
  constexpr int PER = HD / 32, KEYS = WarpState<HD, MAXG>::KEYS;
  const int lane = threadIdx.x & 31;
  const int group = A.q_heads / A.kv_heads;
  const int seq_idx = b / A.T;
  // no __restrict__ here: inside a step kernel q and the newest cache row were written by an earlier phase of the
  // same kernel, and a read-only (non-coherent) load could return what the line held before
  const __nv_bfloat16* kbase = A.kc + ((long long)seq_idx * A.kv_heads + kvh) * A.max_seq * HD + lane * PER;
  const __nv_bfloat16* vbase = A.vc + ((long long)seq_idx * A.kv_heads + kvh) * A.max_seq * HD + lane * PER;
  float qv[MAXG][PER];                                // query vectors of the group, scaled
#pragma unroll
  for (int g = 0; g < MAXG; ++g) {
    Raw<PER> r = {};
    if (g < group) r = load_raw<PER, ONE_BY_ONE>(A.q + ((long long)b * A.q_heads + kvh * group + g) * HD + lane * PER);
    widen<PER>(r, qv[g]);
#pragma unroll
    for (int i = 0; i < PER; ++i) qv[g][i] *= A.scale;
  }
  st.m = -CUDART_INF_F;
  st.l = 0.f;
#pragma unroll
  for (int g = 0; g < MAXG; ++g)
#pragma unroll
    for (int i = 0; i < PER; ++i) st.acc[g][i] = 0.f;
  const int my = lane >> 1;                           // the (key, head) whose score this lane holds
  const int my_key = my / MAXG;
  for (int j = lo + gw * KEYS; j < hi; j += warps * KEYS) {
    Raw<PER> kr[KEYS], vr[KEYS];
#pragma unroll
    for (int k = 0; k < KEYS; ++k) {
      const long long at = (long long)min(j + k, hi - 1) * HD;
      kr[k] = load_raw<PER, ONE_BY_ONE>(kbase + at);
      vr[k] = load_raw<PER, ONE_BY_ONE>(vbase + at);
    }
    float s[16];
#pragma unroll
    for (int k = 0; k < KEYS; ++k) {
      float kf[PER];
      widen<PER>(kr[k], kf);
#pragma unroll
      for (int g = 0; g < MAXG; ++g) {
        float t = 0.f;
#pragma unroll
        for (int i = 0; i < PER; ++i) t += qv[g][i] * kf[i];
        s[k * MAXG + g] = t;
      }
    }
    // after the step with offset o a lane keeps the half of its values that its bit o names
#pragma unroll
    for (int o = 16, n = 8; o > 1; o >>= 1, n >>= 1) {
      const bool up = (lane & o) != 0;
#pragma unroll
      for (int i = 0; i < n; ++i) {
        const float send = up ? s[i] : s[i + n], keep = up ? s[i + n] : s[i];
        s[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
      }
    }
    float sc = s[0] + __shfl_xor_sync(0xffffffffu, s[0], 1);
    if (j + my_key >= hi) sc = -CUDART_INF_F;
    float mx = sc;                                    // over the keys of this head
#pragma unroll
    for (int o = 16; o >= 2 * MAXG; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    const float mn = fmaxf(st.m, mx);                 // finite: key j exists
    const float corr = __expf(st.m - mn), w = __expf(sc - mn);
    float ws = w;
#pragma unroll
    for (int o = 16; o >= 2 * MAXG; o >>= 1) ws += __shfl_xor_sync(0xffffffffu, ws, o);
    st.l = st.l * corr + ws;
    st.m = mn;
#pragma unroll
    for (int g = 0; g < MAXG; ++g) {
      const float cg = __shfl_sync(0xffffffffu, corr, 2 * g);
#pragma unroll
      for (int i = 0; i < PER; ++i) st.acc[g][i] *= cg;
    }
#pragma unroll
    for (int k = 0; k < KEYS; ++k) {
      float vf[PER];
      widen<PER>(vr[k], vf);
#pragma unroll
      for (int g = 0; g < MAXG; ++g) {
        const float wg = __shfl_sync(0xffffffffu, w, 2 * (k * MAXG + g));
#pragma unroll
        for (int i = 0; i < PER; ++i) st.acc[g][i] += wg * vf[i];
      }
    }
  }
  // A maximum ignores NaN, so a warp that saw nothing else would count as one that saw nothing: an infinite maximum makes every
  // merge NaN (weights of the others 0, its own inf - inf).  Decided here, once; in the merges it cost 1.1 of 6.1 us.
  if (st.l != st.l) st.m = CUDART_INF_F;
}

// The keys query token b sees: [lo, hi).
__device__ __forceinline__ void visible(const AttArgs& A, int b, int& lo, int& hi) {
  const int seq_idx = b / A.T;
  const int p = A.pos[seq_idx] + (b - seq_idx * A.T);
  lo = (A.window > 0) ? max(0, p - A.window + 1) : 0;
  hi = p + 1;
}

// One work item (split, kv head, sequence-token b) of the attention; `sm_acc_raw`: ATT_WARPS * group * HD floats of
// shared memory.  The ATT_THREADS computing threads call it together (`sync` is their barrier).
template <int HD, int MAXG, class Sync = AttBlockSync>
__device__ __forceinline__ void attention_item(const AttArgs& A, int split, int kvh, int b, float* sm_acc_raw,
                                               Sync sync = Sync{}) {
  constexpr int PER = HD / 32;
  constexpr int MAX_GROUP = MAXG;
  __nv_bfloat16* out = A.out;
  float* scratch = A.scratch;
  int* counters = A.counters;
  const int q_heads = A.q_heads, kv_heads = A.kv_heads, splits = A.splits;
  const int group = q_heads / kv_heads;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int lo_all, hi_all;
  visible(A, b, lo_all, hi_all);
  const int per_split = (hi_all - lo_all + splits - 1) / splits;
  const int lo = lo_all + split * per_split;
  WarpState<HD, MAXG> st;
  if (A.unaligned) scan_keys<HD, MAXG, true>(A, kvh, b, lo, min(hi_all, lo + per_split), warp, ATT_WARPS, st);
  else scan_keys<HD, MAXG, false>(A, kvh, b, lo, min(hi_all, lo + per_split), warp, ATT_WARPS, st);
  // ---- merge the 8 warps of the CTA through shared memory
  __shared__ float sm_m[ATT_WARPS][MAX_GROUP], sm_l[ATT_WARPS][MAX_GROUP];
  auto sm_acc = [&](int w, int g, int d) -> float& { return sm_acc_raw[((long long)w * group + g) * HD + d]; };
#pragma unroll
  for (int g = 0; g < MAX_GROUP; ++g) {
    if (g < group) {
      if (lane == 2 * g) { sm_m[warp][g] = st.m; sm_l[warp][g] = st.l; }
#pragma unroll
      for (int i = 0; i < PER; ++i) sm_acc(warp, g, lane * PER + i) = st.acc[g][i];
    }
  }
  sync();
  // thread -> (head g, dims d, d + 256/..): 256 threads cover HD dims for one head at a time
  float* part = scratch + (((long long)b * q_heads + kvh * group) * splits + split) * (HD + 2);
  for (int g = 0; g < group; ++g) {
    float mm = -CUDART_INF_F;
#pragma unroll
    for (int w = 0; w < ATT_WARPS; ++w) mm = fmaxf(mm, sm_m[w][g]);
    float ll = 0.f;
#pragma unroll
    for (int w = 0; w < ATT_WARPS; ++w) ll += (sm_m[w][g] == -CUDART_INF_F) ? 0.f : sm_l[w][g] * __expf(sm_m[w][g] - mm);
    float* pg = part + (long long)g * splits * (HD + 2);
    for (int d = threadIdx.x; d < HD; d += ATT_THREADS) {
      float a = 0.f;
#pragma unroll
      for (int w = 0; w < ATT_WARPS; ++w)
        a += (sm_m[w][g] == -CUDART_INF_F) ? 0.f : sm_acc(w, g, d) * __expf(sm_m[w][g] - mm);
      pg[d] = a;
    }
    if (threadIdx.x == 0) { pg[HD] = mm; pg[HD + 1] = ll; }
  }
  // ---- the last CTA of this (sequence, kv head) merges the splits
  __shared__ int is_last;
  __threadfence();
  sync();
  if (threadIdx.x == 0) {
    const int done = atomicAdd(&counters[b * kv_heads + kvh], 1);
    is_last = (done == splits - 1);
    if (is_last) counters[b * kv_heads + kvh] = 0;      // ready for the next launch
  }
  sync();
  if (!is_last) return;
  __threadfence();
  // weights of every (head, split) first — 64 independent loads at most — then the value sums
  // run over independent loads too (no load -> branch -> load chains through L2)
  __shared__ float w_s[MAX_GROUP][64];
  __shared__ float inv_s[MAX_GROUP];
  const float* pbase = scratch + (((long long)b * q_heads + kvh * group) * splits) * (HD + 2);
  for (int idx = threadIdx.x; idx < group * splits; idx += ATT_THREADS) {
    const int g = idx / splits, s = idx % splits;
    w_s[g][s] = __ldcg(pbase + ((long long)g * splits + s) * (HD + 2) + HD);          // m of the split
  }
  sync();
  if ((int)threadIdx.x < group) {
    const int g = threadIdx.x;
    float mm = -CUDART_INF_F;
    for (int s = 0; s < splits; ++s) mm = fmaxf(mm, w_s[g][s]);
    float ll = 0.f;
    for (int s = 0; s < splits; ++s) {
      const float ms = w_s[g][s];
      const float wgt = (ms == -CUDART_INF_F) ? 0.f : __expf(ms - mm);
      ll += wgt * __ldcg(pbase + ((long long)g * splits + s) * (HD + 2) + HD + 1);
      w_s[g][s] = wgt;
    }
    inv_s[g] = ll == 0.f ? 0.f : 1.f / ll;
  }
  sync();
  for (int idx = threadIdx.x; idx < group * HD; idx += ATT_THREADS) {
    const int g = idx / HD, d = idx % HD;
    const float* pg = pbase + (long long)g * splits * (HD + 2) + d;
    float a = 0.f;
#pragma unroll 8
    for (int s = 0; s < splits; ++s) a += __ldcg(pg + (long long)s * (HD + 2)) * w_s[g][s];
    out[((long long)b * q_heads + kvh * group + g) * HD + d] = __float2bfloat16_rn(a * inv_s[g]);
  }
}

}  // namespace decode_att
}  // namespace mesh
