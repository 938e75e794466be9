// Stand-alone launch of the decode-time attention (the work itself: decode_attention.cuh).
#include "decode_attention.cuh"
#include "../device/ptx.cuh"

namespace mesh {
namespace decode_att {

// One token of one sequence is a latency, not a throughput: the keys of a (sequence, KV head) go to the warps of a
// cluster of CTAs, whose partial results meet in shared memory - no scratch in global memory, no fence, no counter, no
// last CTA that finds out that it is the last.  Every CTA merges a slice of the output.
//
// Measured at 700 keys, 8 query heads of 256 over 2 KV heads, back to back: batch 1 17.1 -> 6.6 us, batch 8 32.0 -> 9.8 us
// (16 splits asked for; the keys and values are 1.4 and 11.5 MB, 0.2 and 1.8 us of HBM).
constexpr int MAX_CLUSTER = 8;

template <int HD, int MAXG>
__global__ void __launch_bounds__(ATT_THREADS, MAXG * HD <= 1024 ? 2 : 1) decode_attention_cluster_kernel(const AttArgs A) {
  extern __shared__ float sm_acc[];                      // [ATT_WARPS][MAXG][HD], then the CTA's sums in [0]
  __shared__ float sm_m[ATT_WARPS][MAXG], sm_l[ATT_WARPS][MAXG], cta_m[MAXG], cta_l[MAXG];
  constexpr int PER = HD / 32;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");     // q and the newest cache row come from the previous kernel
  const int ranks = gridDim.x, rank = blockIdx.x, kvh = blockIdx.y, b = blockIdx.z;
  const int group = A.q_heads / A.kv_heads;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int lo, hi;
  visible(A, b, lo, hi);
  WarpState<HD, MAXG> st;
  // neighbouring keys to different CTAs, so that a short context uses all of them
  scan_keys<HD, MAXG, false>(A, kvh, b, lo, hi, warp * ranks + rank, ATT_WARPS * ranks, st);
  if (lane < 2 * MAXG && !(lane & 1)) {
    sm_m[warp][lane >> 1] = st.m;
    sm_l[warp][lane >> 1] = st.l;
  }
#pragma unroll
  for (int g = 0; g < MAXG; ++g)
#pragma unroll
    for (int i = 0; i < PER; ++i) sm_acc[((long long)warp * MAXG + g) * HD + lane * PER + i] = st.acc[g][i];
  __syncthreads();
  // the CTA's sums; a warp that saw no key has m = -inf and weight 0
  constexpr int OUTS = MAXG * HD / ATT_THREADS > 0 ? MAXG * HD / ATT_THREADS : 1;
  float mine[OUTS];
#pragma unroll
  for (int o = 0; o < OUTS; ++o) {
    const int e = threadIdx.x + o * ATT_THREADS;
    if (e < MAXG * HD) {
      const int g = e / HD;
      float mm = -CUDART_INF_F;
#pragma unroll
      for (int w = 0; w < ATT_WARPS; ++w) mm = fmaxf(mm, sm_m[w][g]);
      float a = 0.f, ll = 0.f;
#pragma unroll
      for (int w = 0; w < ATT_WARPS; ++w) {
        const float wgt = sm_m[w][g] == -CUDART_INF_F ? 0.f : __expf(sm_m[w][g] - mm);
        a += wgt * sm_acc[(long long)w * MAXG * HD + e];
        ll += wgt * sm_l[w][g];
      }
      mine[o] = a;
      if (e % HD == 0) { cta_m[g] = mm; cta_l[g] = ll; }
    }
  }
  __syncthreads();
#pragma unroll
  for (int o = 0; o < OUTS; ++o)
    if (threadIdx.x + o * ATT_THREADS < MAXG * HD) sm_acc[threadIdx.x + o * ATT_THREADS] = mine[o];
  cluster_sync_all();
  const int total = group * HD, slice = (total + ranks - 1) / ranks;
  for (int e = rank * slice + threadIdx.x; e < min(total, (rank + 1) * slice); e += ATT_THREADS) {
    const int g = e / HD;
    float m[MAX_CLUSTER], l[MAX_CLUSTER], v[MAX_CLUSTER];
#pragma unroll
    for (int r = 0; r < MAX_CLUSTER; ++r) {
      m[r] = -CUDART_INF_F;
      if (r < ranks) {
        asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(m[r]) : "r"(mapa_u32(smem_u32(&cta_m[g]), r)));
        asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(l[r]) : "r"(mapa_u32(smem_u32(&cta_l[g]), r)));
        asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v[r]) : "r"(mapa_u32(smem_u32(sm_acc + e), r)));
      }
    }
    float mm = -CUDART_INF_F;
#pragma unroll
    for (int r = 0; r < MAX_CLUSTER; ++r) mm = fmaxf(mm, m[r]);
    float a = 0.f, ll = 0.f;
#pragma unroll
    for (int r = 0; r < MAX_CLUSTER; ++r) {
      const float wgt = m[r] == -CUDART_INF_F ? 0.f : __expf(m[r] - mm);
      if (wgt != 0.f) { a += wgt * v[r]; ll += wgt * l[r]; }
    }
    A.out[((long long)b * A.q_heads + kvh * group) * HD + e] = __float2bfloat16_rn(ll == 0.f ? 0.f : a / ll);
  }
  cluster_sync_all();                                    // nobody's shared memory goes away while it is read
}

// Many splits of a long context, and inputs that vector loads do not take: partial results in global memory, merged by the CTA
// that finishes last.
// Grid = (splits, kv_heads, batch * tokens): one work item per CTA.
template <int HD, int MAXG>
__global__ void __launch_bounds__(ATT_THREADS) decode_attention_kernel(const AttArgs A) {
  extern __shared__ float sm_acc[];                      // [ATT_WARPS][group][HD]
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  attention_item<HD, MAXG>(A, blockIdx.x, blockIdx.y, blockIdx.z, sm_acc);
}

template <int HD, int MAXG>
static int launch(const AttArgs& A, bool cluster, void* stream) {
  void (*kern)(const AttArgs) = cluster ? decode_attention_cluster_kernel<HD, MAXG> : decode_attention_kernel<HD, MAXG>;
  const size_t smem = (size_t)ATT_WARPS * MAXG * HD * sizeof(float);
  static bool configured[2] = {false, false};
  if (smem > 32 * 1024 && !configured[cluster]) {        // with the static arrays above the default limit
    MESH_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    configured[cluster] = true;
  }
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  unsigned x = A.splits;
  if (cluster) x = x >= 8 ? 8 : x >= 4 ? 4 : x >= 2 ? 2 : 1;
  cfg.gridDim = dim3(x, A.kv_heads, A.B * A.T);
  cfg.blockDim = dim3(ATT_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = (cudaStream_t)stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = pdl_enabled() ? 1 : 0;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = x;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = cluster ? 2 : 1;
  MESH_CUDA_OK(cudaLaunchKernelEx(&cfg, kern, A));
  MESH_CUDA_OK(cudaGetLastError());
  return 0;
}

}  // namespace decode_att
}  // namespace mesh


extern "C" int mesh_decode_attention_scratch_floats(int B, int q_heads, int head_dim, int splits) {
  return B * q_heads * splits * (head_dim + 2);
}

extern "C" int mesh_decode_attention(const void* q, const void* k_cache, const void* v_cache, const int* pos, void* out,
                                     float* scratch, int* counters, int B, int tokens_per_seq, int q_heads, int kv_heads,
                                     int head_dim, int max_seq, int window, float scale, int splits, void* stream) {
  using namespace mesh;
  using namespace mesh::decode_att;
  if (B <= 0) return 0;
  if (q_heads % kv_heads || q_heads / kv_heads > MAX_GROUPS) return set_error(-2, "decode_attention: group size must be 1..8");
  if (splits < 1 || splits > 64) return set_error(-2, "decode_attention: splits must be 1..64");
  if (tokens_per_seq < 1) tokens_per_seq = 1;
  AttArgs A;
  memset(&A, 0, sizeof(A));
  A.q = (const __nv_bfloat16*)q; A.kc = (const __nv_bfloat16*)k_cache; A.vc = (const __nv_bfloat16*)v_cache; A.pos = pos;
  A.out = (__nv_bfloat16*)out; A.scratch = scratch; A.counters = counters;
  A.q_heads = q_heads; A.kv_heads = kv_heads; A.max_seq = max_seq; A.window = window; A.scale = scale; A.splits = splits;
  A.T = tokens_per_seq; A.B = B; A.head_dim = head_dim;
  A.unaligned = unaligned(q, k_cache, v_cache, head_dim);
  // A cluster, or splits merged through memory.  The host knows the size of the cache and not the context, so the line lies where
  // a full cache takes as long either way.  Back to back, 8 query heads of 256 over 2 KV heads, batch 1 / 8, a cluster of eight
  // and 16 splits: at 4096 keys 18.5 / 29.0 and 19.1 / 26.2 us, at 8192 32.1 / 56.3 and 25.5 / 40.3, at 200 keys of a cache of
  // 8192 5.1 / 6.6 and 11.4 / 12.4; 32 heads of 128 over 8, 4096 keys 15.1 / 47.5 and 19.0 / 54.4, 8192 25.5 / 85.0 and
  // 26.6 / 80.3.  Whoever asks for no more splits than a cluster has CTAs gets the cluster.
  const int most = window > 0 && window < max_seq ? window : max_seq;
  const bool cluster = !A.unaligned && (splits <= MAX_CLUSTER || most <= 4096);
  const bool four = q_heads / kv_heads <= 4;
  switch (head_dim) {
    case 256: return four ? launch<256, 4>(A, cluster, stream) : launch<256, 8>(A, cluster, stream);
    case 128: return four ? launch<128, 4>(A, cluster, stream) : launch<128, 8>(A, cluster, stream);
    case 64: return four ? launch<64, 4>(A, cluster, stream) : launch<64, 8>(A, cluster, stream);
    default: return set_error(-2, "decode_attention: head_dim must be 64, 128 or 256");
  }
}
