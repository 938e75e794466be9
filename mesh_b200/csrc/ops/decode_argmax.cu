// Vocabulary-parallel greedy selection: a CTA, or a cluster of them, per sequence finds (max logit, lowest index) over this
// rank's vocabulary shard (a slice each, the pairs meet in the first CTA's shared memory), exchanges that 8-byte pair with
// every rank, and all ranks pick the same winner (highest value, lowest global index on ties) without ever gathering logits.
#include <cuda_runtime.h>
#include <math_constants.h>
#include "decode_api.h"
#include "../device/ptx.cuh"
#include "../runtime/host_common.h"
#include <cstring>

namespace mesh {
namespace {

constexpr int AM_THREADS = 1024;
// One CTA of 1024 threads is a chain of loads over a long vocabulary, and a cluster's barriers cost more than a short one.
// Back to back at batch 1 / 8, one CTA and eight: 4096 logits 1.7 / 1.8 and 2.2 / 2.4 us, 16384 2.0 / 2.2 and 2.2 / 2.6,
// 32768 2.5 / 2.6 and 2.3 / 2.8, 65536 3.4 / 3.6 and 2.6 / 3.0, 262144 8.7 / 8.9 and 3.2 / 3.9.
constexpr int MOST_CTAS = 8, ONE_CTA_VOCAB = 16384;

__device__ __forceinline__ void better(float& v, int& i, float ov, int oi) {
  if (ov > v || (ov == v && oi < i)) { v = ov; i = oi; }
}

template <int AM_CTAS>
__global__ void __launch_bounds__(AM_THREADS)
decode_argmax_kernel(const float* __restrict__ logits, long long ldl, int vocab_local, int vocab_offset,
                     int* __restrict__ tokens_out, int* __restrict__ pos, int rank, int world,
                     uint2* const* __restrict__ xchg_unused, uint2* x0, uint2* x1, uint2* x2, uint2* x3, uint2* x4,
                     uint2* x5, uint2* x6, uint2* x7, uint32_t* step, Status* st) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (AM_CTAS > 1) cluster_arrive_relaxed();             // waited for before the store into the first CTA's shared memory
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int b = blockIdx.x / AM_CTAS, part = blockIdx.x % AM_CTAS;
  const uint32_t seq = (step ? *step : 0u) + 1u;
  const float* row = logits + (long long)b * ldl;
  float best = -CUDART_INF_F;
  int bi = 0x7fffffff;
  const int per = ((vocab_local + AM_CTAS - 1) / AM_CTAS + 3) & ~3;
  const int lo = part * per, hi = min(vocab_local, lo + per);
  int i = lo + threadIdx.x * 4;
  if ((reinterpret_cast<uintptr_t>(row) & 15) == 0) {
#pragma unroll 4
    for (; i + 4 <= hi; i += AM_THREADS * 4) {       // ascending per thread: the first maximum is kept
      const float4 v = *reinterpret_cast<const float4*>(row + i);
      if (v.x > best) { best = v.x; bi = i; }
      if (v.y > best) { best = v.y; bi = i + 1; }
      if (v.z > best) { best = v.z; bi = i + 2; }
      if (v.w > best) { best = v.w; bi = i + 3; }
    }
  }
  for (; i < hi; i += AM_THREADS * 4)
    for (int e = i; e < min(i + 4, hi); ++e)
      if (row[e] > best) { best = row[e]; bi = e; }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, best, o);
    const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
    better(best, bi, ov, oi);
  }
  __shared__ float sv[32];
  __shared__ int si[32];
  __shared__ float pv[AM_CTAS];
  __shared__ int pi[AM_CTAS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) { sv[warp] = best; si[warp] = bi; }
  __syncthreads();
  if (AM_CTAS > 1) cluster_wait();
  if (warp == 0) {
    best = sv[lane];
    bi = si[lane];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      better(best, bi, ov, oi);
    }
    if (AM_CTAS > 1 && lane == 0) {
      asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(mapa_u32(smem_u32(&pv[part]), 0)), "f"(best) : "memory");
      asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(mapa_u32(smem_u32(&pi[part]), 0)), "r"(bi) : "memory");
    }
    __syncwarp();
  }
  if (AM_CTAS > 1) cluster_sync_all();
  if (part != 0 || warp != 0) return;
  if (AM_CTAS > 1) {
    best = lane < AM_CTAS ? pv[lane] : -CUDART_INF_F;
    bi = lane < AM_CTAS ? pi[lane] : 0x7fffffff;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      better(best, bi, ov, oi);
    }
  }
  int gidx = bi + vocab_offset;
  if (world > 1) {
    uint2* peers[8] = {x0, x1, x2, x3, x4, x5, x6, x7};
    // slot layout on every rank: [parity(seq & 1)][src rank][sequence][2 words]: {value bits, seq}, {index, seq}
    const long long base = ((long long)(seq & 1u) * world * 8 + (long long)rank * 8 + b) * 2;
    if (lane < world) {
      uint2* p = peers[lane] + base;
      asm volatile("st.volatile.global.v2.u32 [%0], {%1, %2};" ::"l"(p), "r"(__float_as_uint(best)), "r"(seq) : "memory");
      asm volatile("st.volatile.global.v2.u32 [%0], {%1, %2};" ::"l"(p + 1), "r"((uint32_t)gidx), "r"(seq) : "memory");
    }
    float v = -CUDART_INF_F;
    int id = 0x7fffffff;
    if (lane < world) {
      const uint2* p = peers[rank] + ((long long)(seq & 1u) * world * 8 + (long long)lane * 8 + b) * 2;
      uint2 w0, w1;
      unsigned long long t0 = 0;
      uint32_t it = 0;
      while (true) {
        asm volatile("ld.volatile.global.v2.u32 {%0, %1}, [%2];" : "=r"(w0.x), "=r"(w0.y) : "l"(p) : "memory");
        asm volatile("ld.volatile.global.v2.u32 {%0, %1}, [%2];" : "=r"(w1.x), "=r"(w1.y) : "l"(p + 1) : "memory");
        if (w0.y == seq && w1.y == seq) break;
        if (((++it) & 0x3ffu) == 0) {
          if (t0 == 0) t0 = globaltimer_ns();
          else if (globaltimer_ns() - t0 > MESH_WAIT_LIMIT_NS || status_aborted(st)) {
            status_record(st, MESH_TIMEOUT, SITE_PEER_FLAG, seq, w0.y, (unsigned long long)p);
            break;
          }
        }
      }
      v = __uint_as_float(w0.x);
      id = (int)w1.x;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, v, o);
      const int oi = __shfl_xor_sync(0xffffffffu, id, o);
      if (ov > v || (ov == v && oi < id)) { v = ov; id = oi; }
    }
    gidx = id;
  }
  if (lane == 0) {
    tokens_out[b] = gidx;
    if (pos) pos[b] += 1;
    // the last sequence's CTA to finish advances the step word (every CTA has read it by then:
    // the counter below is only bumped after this CTA's own read at the top)
    if (step) {
      __threadfence();
      const unsigned done = atomicAdd(step + 1, 1u);
      if (done == gridDim.x / AM_CTAS - 1) { step[1] = 0; __threadfence(); atomicAdd(step, 1u); }
    }
  }
}

}  // namespace
}  // namespace mesh

extern "C" int mesh_decode_argmax(const float* logits, long long ldl, int B, int vocab_local, int vocab_offset,
                                  int* tokens_out, int* pos, int rank, int world, void* const* xchg, uint32_t* step,
                                  void* status, void* stream) {
  using namespace mesh;
  if (B < 1 || B > 8) return set_error(-2, "decode_argmax: batch must be 1..8");
  if (world < 1 || world > 8) return set_error(-4, "decode_argmax: world out of range");
  uint2* x[8] = {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr};
  for (int r = 0; r < world && xchg; ++r) x[r] = (uint2*)xchg[r];
  const int ctas = vocab_local <= ONE_CTA_VOCAB ? 1 : MOST_CTAS;
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3((unsigned)(B * ctas));
  cfg.blockDim = dim3(AM_THREADS);
  cfg.stream = (cudaStream_t)stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = pdl_enabled() ? 1 : 0;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = (unsigned)ctas;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = ctas > 1 ? 2 : 1;
  uint2* const* none = nullptr;
  MESH_CUDA_OK(cudaLaunchKernelEx(&cfg, ctas > 1 ? decode_argmax_kernel<MOST_CTAS> : decode_argmax_kernel<1>, logits, ldl, vocab_local, vocab_offset, tokens_out, pos, rank,
                                  world, none, x[0], x[1], x[2], x[3], x[4], x[5], x[6], x[7], step, (Status*)status));
  return 0;
}
