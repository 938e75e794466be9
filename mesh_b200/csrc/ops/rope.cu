// Rotate-half rotary position embedding, in place, bf16 activations with fp32 cos/sin tables.
// Reference model: examples/pl.py:17-28 (cached cos/sin, rotate-half); theta is folded into the
// tables by the caller (1e6 for the E2B-class config).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include "ops_api.h"
#include "../runtime/host_common.h"

namespace mesh {
namespace {

// One thread rotates 8 consecutive pairs (i, i + hd/2): two 16-byte loads, two 16-byte stores.
__global__ void rope_kernel(__nv_bfloat16* __restrict__ x, const int* __restrict__ pos,
                            const float* __restrict__ cos_t, const float* __restrict__ sin_t, int tokens,
                            int heads, int hd, long long ld, int inverse) {
  const int half = hd >> 1;
  const int vec_per_head = half >> 3;
  const long long total = (long long)tokens * heads * vec_per_head;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const int v = (int)(idx % vec_per_head);
    const int h = (int)((idx / vec_per_head) % heads);
    const int t = (int)(idx / ((long long)vec_per_head * heads));
    const int p = pos[t];
    __nv_bfloat16* base = x + (long long)t * ld + (long long)h * hd + v * 8;
    uint4 lo = *reinterpret_cast<uint4*>(base);
    uint4 hi = *reinterpret_cast<uint4*>(base + half);
    const float4* c4 = reinterpret_cast<const float4*>(cos_t + (long long)p * half + v * 8);
    const float4* s4 = reinterpret_cast<const float4*>(sin_t + (long long)p * half + v * 8);
    float c[8], s[8];
    *reinterpret_cast<float4*>(c) = c4[0];
    *reinterpret_cast<float4*>(c + 4) = c4[1];
    *reinterpret_cast<float4*>(s) = s4[0];
    *reinterpret_cast<float4*>(s + 4) = s4[1];
    __nv_bfloat162* l2 = reinterpret_cast<__nv_bfloat162*>(&lo);
    __nv_bfloat162* h2 = reinterpret_cast<__nv_bfloat162*>(&hi);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float2 a = __bfloat1622float2(l2[i]);
      float2 b = __bfloat1622float2(h2[i]);
      const float s0 = inverse ? -s[2 * i] : s[2 * i], s1 = inverse ? -s[2 * i + 1] : s[2 * i + 1];
      float2 oa, ob;
      oa.x = a.x * c[2 * i] - b.x * s0;
      ob.x = b.x * c[2 * i] + a.x * s0;
      oa.y = a.y * c[2 * i + 1] - b.y * s1;
      ob.y = b.y * c[2 * i + 1] + a.y * s1;
      l2[i] = __floats2bfloat162_rn(oa.x, oa.y);
      h2[i] = __floats2bfloat162_rn(ob.x, ob.y);
    }
    *reinterpret_cast<uint4*>(base) = lo;
    *reinterpret_cast<uint4*>(base + half) = hi;
  }
}

// Eight pairs (i, i + hd / 2) rotated by +- their angles.
__device__ __forceinline__ void rotate8(float (&a)[8], float (&b)[8], const float* __restrict__ cos_t, const float* __restrict__ sin_t,
                                        float sign) {
  float c[8], s[8];
  *reinterpret_cast<float4*>(c) = __ldg(reinterpret_cast<const float4*>(cos_t));
  *reinterpret_cast<float4*>(c + 4) = __ldg(reinterpret_cast<const float4*>(cos_t) + 1);
  *reinterpret_cast<float4*>(s) = __ldg(reinterpret_cast<const float4*>(sin_t));
  *reinterpret_cast<float4*>(s + 4) = __ldg(reinterpret_cast<const float4*>(sin_t) + 1);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float x = a[i], y = b[i], sn = sign * s[i];
    a[i] = x * c[i] - y * sn;
    b[i] = y * c[i] + x * sn;
  }
}
__device__ __forceinline__ void load8(const __nv_bfloat16* p, float (&f)[8]) {
  const uint4 q = *reinterpret_cast<const uint4*>(p);
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&q);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 t = __bfloat1622float2(h[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}
__device__ __forceinline__ void store8(__nv_bfloat16* p, const float (&f)[8]) {
  uint4 q;
  __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&q);
#pragma unroll
  for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  *reinterpret_cast<uint4*>(p) = q;
}

// The fused projection [tokens, (q_heads + 2 kv_heads) * HD] copied with its query and key heads rotated.  A thread takes
// eight pairs of one head.
template <int HD>
__global__ void __launch_bounds__(256) rope_qkv_kernel(const __nv_bfloat16* __restrict__ src, long long ld, __nv_bfloat16* __restrict__ dst,
                                                       const int* __restrict__ pos, const float* __restrict__ cos_t,
                                                       const float* __restrict__ sin_t, int tokens, int heads, int rotated) {
  constexpr int HALF = HD / 2, VPH = HALF / 8;
  const long long total = (long long)tokens * heads * VPH;
  for (long long idx = blockIdx.x * 256ll + threadIdx.x; idx < total; idx += gridDim.x * 256ll) {
    const int v = (int)(idx % VPH);
    const long long th = idx / VPH;
    const int h = (int)(th % heads);
    const long long t = th / heads;
    const __nv_bfloat16* in = src + t * ld + h * HD + v * 8;
    __nv_bfloat16* out = dst + th * HD + v * 8;
    if (h < rotated) {
      const long long at = (long long)pos[t] * HALF + v * 8;
      float a[8], b[8];
      load8(in, a);
      load8(in + HALF, b);
      rotate8(a, b, cos_t + at, sin_t + at, 1.f);
      store8(out, a);
      store8(out + HALF, b);
    } else {
      *reinterpret_cast<uint4*>(out) = *reinterpret_cast<const uint4*>(in);
      *reinterpret_cast<uint4*>(out + HALF) = *reinterpret_cast<const uint4*>(in + HALF);
    }
  }
}

// Its gradient: the query columns from the fp32 accumulator dq [tokens, q_heads * HD], the key columns in place.
template <int HD>
__global__ void __launch_bounds__(256) rope_qkv_bwd_kernel(const float* __restrict__ dq, __nv_bfloat16* __restrict__ d,
                                                           const int* __restrict__ pos, const float* __restrict__ cos_t,
                                                           const float* __restrict__ sin_t, int tokens, int q_heads, int rotated, int heads) {
  constexpr int HALF = HD / 2, VPH = HALF / 8;
  const long long total = (long long)tokens * rotated * VPH;
  for (long long idx = blockIdx.x * 256ll + threadIdx.x; idx < total; idx += gridDim.x * 256ll) {
    const int v = (int)(idx % VPH);
    const long long th = idx / VPH;
    const int h = (int)(th % rotated);
    const long long t = th / rotated;
    __nv_bfloat16* out = d + (t * heads + h) * HD + v * 8;
    float a[8], b[8];
    if (h < q_heads) {
      const float* in = dq + (t * q_heads + h) * HD + v * 8;
      *reinterpret_cast<float4*>(a) = __ldg(reinterpret_cast<const float4*>(in));
      *reinterpret_cast<float4*>(a + 4) = __ldg(reinterpret_cast<const float4*>(in) + 1);
      *reinterpret_cast<float4*>(b) = __ldg(reinterpret_cast<const float4*>(in + HALF));
      *reinterpret_cast<float4*>(b + 4) = __ldg(reinterpret_cast<const float4*>(in + HALF) + 1);
    } else {
      load8(out, a);
      load8(out + HALF, b);
    }
    const long long at = (long long)pos[t] * HALF + v * 8;
    rotate8(a, b, cos_t + at, sin_t + at, -1.f);
    store8(out, a);
    store8(out + HALF, b);
  }
}

}  // namespace
}  // namespace mesh

extern "C" int mesh_rope_qkv(const void* src, long long ld, void* dst, const int* positions, const float* cos_t, const float* sin_t,
                             int tokens, int q_heads, int kv_heads, int head_dim, void* stream) {
  using namespace mesh;
  const int heads = q_heads + 2 * kv_heads;
  if (tokens <= 0 || heads <= 0) return 0;
  if (ld % 8 || (uintptr_t)src % 16 || (uintptr_t)dst % 16) return set_error(-2, "rope_qkv: rows must be 16-byte aligned");
  const long long total = (long long)tokens * heads * (head_dim / 16);
  const unsigned grid = (unsigned)((total + 255) / 256 < 148 * 16 ? (total + 255) / 256 : 148 * 16);
#define MESH_ROPE(HD)                                                                                                             \
  rope_qkv_kernel<HD><<<grid, 256, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)src, ld, (__nv_bfloat16*)dst, positions, cos_t, \
                                                              sin_t, tokens, heads, q_heads + kv_heads)
  switch (head_dim) {
    case 64: MESH_ROPE(64); break;
    case 128: MESH_ROPE(128); break;
    case 256: MESH_ROPE(256); break;
    default: return set_error(-2, "rope_qkv: head_dim must be 64, 128 or 256");
  }
#undef MESH_ROPE
  MESH_CUDA_OK(cudaGetLastError());
  return 0;
}

extern "C" int mesh_rope_qkv_bwd(const float* dq, void* dqkv, const int* positions, const float* cos_t, const float* sin_t, int tokens,
                                 int q_heads, int kv_heads, int head_dim, void* stream) {
  using namespace mesh;
  if (tokens <= 0 || q_heads + kv_heads <= 0) return 0;
  if ((uintptr_t)dq % 16 || (uintptr_t)dqkv % 16) return set_error(-2, "rope_qkv_bwd: rows must be 16-byte aligned");
  const long long total = (long long)tokens * (q_heads + kv_heads) * (head_dim / 16);
  const unsigned grid = (unsigned)((total + 255) / 256 < 148 * 16 ? (total + 255) / 256 : 148 * 16);
#define MESH_ROPE(HD)                                                                                                                \
  rope_qkv_bwd_kernel<HD><<<grid, 256, 0, (cudaStream_t)stream>>>(dq, (__nv_bfloat16*)dqkv, positions, cos_t, sin_t, tokens, q_heads, \
                                                                  q_heads + kv_heads, q_heads + 2 * kv_heads)
  switch (head_dim) {
    case 64: MESH_ROPE(64); break;
    case 128: MESH_ROPE(128); break;
    case 256: MESH_ROPE(256); break;
    default: return set_error(-2, "rope_qkv_bwd: head_dim must be 64, 128 or 256");
  }
#undef MESH_ROPE
  MESH_CUDA_OK(cudaGetLastError());
  return 0;
}

extern "C" int mesh_rope(void* x, const int* positions, const float* cos_t, const float* sin_t, int tokens, int heads,
                         int head_dim, long long ld, int inverse, void* stream) {
  using namespace mesh;
  if (tokens <= 0 || heads <= 0) return 0;
  if (head_dim % 16 || ld % 8) return set_error(-2, "rope: head_dim must be a multiple of 16 and ld of 8");
  const long long total = (long long)tokens * heads * (head_dim / 16);
  int grid = (int)((total + 255) / 256);
  if (grid > 148 * 16) grid = 148 * 16;
  rope_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>((__nv_bfloat16*)x, positions, cos_t, sin_t, tokens, heads,
                                                      head_dim, ld, inverse);
  MESH_CUDA_OK(cudaGetLastError());
  return 0;
}
