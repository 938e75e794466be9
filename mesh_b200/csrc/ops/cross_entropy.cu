// Cross-entropy over a vocabulary shard: the per-row statistics in one pass over the logits, and the gradient in one.
//
// With the output projection column-parallel a rank holds logits[:, v0:v1].  The loss of a row needs the row's
// maximum, its sum of exponentials and the target's logit over the WHOLE vocabulary; each rank computes them over its
// columns here (online max / sum, the reference's statistics of compiler/mesh_compiler/operations.py:6281-6330), two
// tiny all-reduces combine them, and the gradient (softmax - onehot) * g is formed from the logits again, so no fp32
// copy of the logits or of their exponentials is ever stored.
//
// Bound by HBM: 8192 rows of 50304 logits (824 MB) are read in 156 us for the statistics (5.3 TB/s; 290 us before the
// exponentials were batched) and read and written in 273 us for the gradient (6.0 TB/s).  Where the whole vocabulary is
// here, losses, their mean and the gradient are these launches and one small one: 641 -> 454 us a call forward and backward,
// some twenty tensor operations on the rows among what went.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math_constants.h>
#include "ops_api.h"
#include "../runtime/host_common.h"

namespace mesh {
namespace {

constexpr int CE_THREADS = 256;
constexpr float LOG2E = 1.4426950408889634f;

__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ void merge(float& m, float& s, float m2, float s2) {
  const float mm = fmaxf(m, m2);
  if (mm == -CUDART_INF_F) { s += s2; return; }       // nothing finite yet: both sums are 0, or NaN from a NaN logit
  s = s * __expf(m - mm) + s2 * __expf(m2 - mm);
  m = mm;
}
__device__ __forceinline__ void unpack8(const uint4& q, float (&f)[8]) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&q);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 t = __bfloat1622float2(h[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}
// 2^((f - m) log2(e)), two at a time.  The maximum is subtracted before the scaling: near it the difference is exact, while
// -m log2(e) as the addend of an fma is rounded in proportion to m (1e-5 of a probability at logits of 1000) and is infinite
// for a mask of bf16's lowest value.
__device__ __forceinline__ void exp_off(float f0, float f1, float m, float& e0, float& e1) {
  unsigned long long v, o;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(f0), "f"(f1));
  asm("mov.b64 %0, {%1, %1};" : "=l"(o) : "f"(-m));
  asm("add.rn.f32x2 %0, %0, %1;" : "+l"(v) : "l"(o));
  asm("mov.b64 %0, {%1, %1};" : "=l"(o) : "f"(LOG2E));
  asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(v) : "l"(o));
  asm("mov.b64 {%0, %1}, %2;" : "=f"(e0), "=f"(e1) : "l"(v));
  e0 = ex2_approx(e0);
  e1 = ex2_approx(e1);
}
// Eight values at a time: one comparison with the running maximum, and the exponentials relative to it in one ex2 each
// (value by value, with a branch and two exponentials in it, the pass ran at 2.8 TB/s).
__device__ __forceinline__ void online8(float& m, float& s, const uint4& q) {
  float f[8];
  unpack8(q, f);
  const float mx = fmaxf(fmaxf(fmaxf(f[0], f[1]), fmaxf(f[2], f[3])), fmaxf(fmaxf(f[4], f[5]), fmaxf(f[6], f[7])));
  if (mx > m) { s *= __expf(m - mx); m = mx; }
  const float ref = (m == -CUDART_INF_F) ? 0.f : m;
  float a = 0.f, b = 0.f;
#pragma unroll
  for (int i = 0; i < 8; i += 2) {
    float e0, e1;
    exp_off(f[i], f[i + 1], ref, e0, e1);
    a += e0;
    b += e1;
  }
  s += a + b;
}
__device__ __forceinline__ void online(float& m, float& s, float x) {
  if (x > m) { s = s * __expf(m - x) + 1.f; m = x; }
  else if (x != -CUDART_INF_F) s += __expf(x - m);    // NaN comes here, also as the first value
}

// Elements of a row before its first 16-byte boundary (rows of an odd width start anywhere).
__device__ __forceinline__ int head_of(const __nv_bfloat16* x, int cols) {
  return min(cols, (int)(((16 - (reinterpret_cast<uintptr_t>(x) & 15)) & 15) >> 1));
}

// row_max[r], row_sum[r] (relative to row_max[r]) and target_logit[r] (0 when the target is not in this shard or ignored).
// `loss` (may be null, the whole vocabulary is here then): the token's loss, 0 when ignored.
__global__ void __launch_bounds__(CE_THREADS)
ce_stats_kernel(const __nv_bfloat16* __restrict__ logits, long long ld, int rows, int cols, const long long* __restrict__ targets,
                long long vocab_start, long long ignore_index, float* __restrict__ row_max, float* __restrict__ row_sum,
                float* __restrict__ target_logit, float* __restrict__ loss) {
  __shared__ float sm[CE_THREADS / 32], ss[CE_THREADS / 32];
  for (int r = blockIdx.x; r < rows; r += gridDim.x) {
    const __nv_bfloat16* x = logits + (long long)r * ld;
    float m = -CUDART_INF_F, s = 0.f;
    const int head = head_of(x, cols);
    const int nv = (cols - head) >> 3;
    const uint4* xv = reinterpret_cast<const uint4*>(x + head);
    int v = threadIdx.x;
    for (; v + 3 * CE_THREADS < nv; v += 4 * CE_THREADS) {             // four loads in flight
      uint4 q[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) q[u] = __ldg(xv + v + u * CE_THREADS);
#pragma unroll
      for (int u = 0; u < 4; ++u) online8(m, s, q[u]);
    }
    for (; v < nv; v += CE_THREADS) online8(m, s, __ldg(xv + v));
    for (int c = threadIdx.x; c < head; c += CE_THREADS) online(m, s, __bfloat162float(x[c]));
    for (int c = head + nv * 8 + threadIdx.x; c < cols; c += CE_THREADS) online(m, s, __bfloat162float(x[c]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float m2 = __shfl_xor_sync(0xffffffffu, m, o), s2 = __shfl_xor_sync(0xffffffffu, s, o);
      merge(m, s, m2, s2);
    }
    if ((threadIdx.x & 31) == 0) { sm[threadIdx.x >> 5] = m; ss[threadIdx.x >> 5] = s; }
    __syncthreads();
    if (threadIdx.x == 0) {
      float M = sm[0], S = ss[0];
      for (int w = 1; w < CE_THREADS / 32; ++w) merge(M, S, sm[w], ss[w]);
      row_max[r] = M;
      row_sum[r] = S;
      const long long t = targets[r], local = t - vocab_start;
      const float tl = (t != ignore_index && local >= 0 && local < cols) ? __bfloat162float(x[local]) : 0.f;
      target_logit[r] = tl;
      if (loss) loss[r] = t != ignore_index ? logf(S) + (M - tl) : 0.f;
    }
    __syncthreads();
  }
}

// out = sum(loss), or that over the number of tokens that are not ignored (at least 1); divisor: what it was divided by.
__global__ void __launch_bounds__(1024)
ce_reduce_kernel(const float* __restrict__ loss, const long long* __restrict__ targets, int rows, long long ignore_index, int mean,
                 float* __restrict__ out, float* __restrict__ divisor) {
  __shared__ float sl[32];
  __shared__ int sn[32];
  float l = 0.f;
  int n = 0;
  for (int i = threadIdx.x; i < rows; i += 1024) {
    l += loss[i];
    n += targets[i] != ignore_index;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    l += __shfl_xor_sync(0xffffffffu, l, o);
    n += __shfl_xor_sync(0xffffffffu, n, o);
  }
  if ((threadIdx.x & 31) == 0) { sl[threadIdx.x >> 5] = l; sn[threadIdx.x >> 5] = n; }
  __syncthreads();
  if (threadIdx.x < 32) {
    l = sl[threadIdx.x];
    n = sn[threadIdx.x];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      l += __shfl_xor_sync(0xffffffffu, l, o);
      n += __shfl_xor_sync(0xffffffffu, n, o);
    }
    if (threadIdx.x == 0) {
      const float div = mean ? (float)max(n, 1) : 1.f;
      *out = l / div;
      *divisor = div;
    }
  }
}

__device__ __forceinline__ uint4 grad8(const uint4& q, float m, float inv) {
  float f[8];
  unpack8(q, f);
  uint4 o;
  __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float e0, e1;
    exp_off(f[2 * i], f[2 * i + 1], m, e0, e1);
    h[i] = __floats2bfloat162_rn(e0 * inv, e1 * inv);
  }
  return o;
}

// d[r, c] = (exp(x - gmax[r]) / gsum[r] - [c == target]) * g / divisor, 0 in ignored rows.  g: one value per row, or one for
// all of them (g_stride 0); divisor: may be null.  The target's element is written once more after the row: no comparison
// per element.
__global__ void __launch_bounds__(CE_THREADS)
ce_grad_kernel(const __nv_bfloat16* __restrict__ logits, long long ld, __nv_bfloat16* d, long long ldd, int rows, int cols,
               const long long* __restrict__ targets, long long vocab_start, long long ignore_index,
               const float* __restrict__ gmax, const float* __restrict__ gsum, const float* __restrict__ gscale, int g_stride,
               const float* __restrict__ divisor) {
  for (int r = blockIdx.x; r < rows; r += gridDim.x) {
    const __nv_bfloat16* x = logits + (long long)r * ld;
    __nv_bfloat16* o = d + (long long)r * ldd;
    const long long t = targets[r], local = t - vocab_start;
    float g = gscale[(long long)r * g_stride];
    if (divisor) g /= divisor[0];
    if (t == ignore_index) g = 0.f;
    const float mx = gmax[r], inv = g / gsum[r];
    const bool mine = local >= 0 && local < cols;
    // d may be the logits themselves: the target's logit is read before its element is written
    const float tx = (threadIdx.x == 0 && mine) ? __bfloat162float(x[local]) : 0.f;
    __syncthreads();
    const bool vec = ((reinterpret_cast<uintptr_t>(x) ^ reinterpret_cast<uintptr_t>(o)) & 15) == 0;
    const int head = vec ? head_of(x, cols) : cols;
    const int nv = (cols - head) >> 3;
    const uint4* xv = reinterpret_cast<const uint4*>(x + head);
    uint4* ov = reinterpret_cast<uint4*>(o + head);
    int v = threadIdx.x;
    for (; v + 3 * CE_THREADS < nv; v += 4 * CE_THREADS) {
      uint4 q[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) q[u] = xv[v + u * CE_THREADS];
#pragma unroll
      for (int u = 0; u < 4; ++u) __stcs(ov + v + u * CE_THREADS, grad8(q[u], mx, inv));
    }
    for (; v < nv; v += CE_THREADS) ov[v] = grad8(xv[v], mx, inv);
    for (int c = threadIdx.x; c < head; c += CE_THREADS) o[c] = __float2bfloat16_rn(__expf(__bfloat162float(x[c]) - mx) * inv);
    for (int c = head + nv * 8 + threadIdx.x; c < cols; c += CE_THREADS)
      o[c] = __float2bfloat16_rn(__expf(__bfloat162float(x[c]) - mx) * inv);
    __syncthreads();
    if (threadIdx.x == 0 && mine) o[local] = __float2bfloat16_rn(__expf(tx - mx) * inv - g);
  }
}

}  // namespace
}  // namespace mesh

extern "C" int mesh_ce_loss_bf16(const void* logits, long long ld, int rows, int cols, const long long* targets,
                                 long long vocab_start, long long ignore_index, float* row_max, float* row_sum,
                                 float* target_logit, float* loss, void* stream) {
  using namespace mesh;
  if (rows <= 0 || cols <= 0) return 0;
  if (!logits || !targets || !row_max || !row_sum || !target_logit) return set_error(-2, "ce_stats: null argument");
  int grid = rows < 148 * 8 ? rows : 148 * 8;
  ce_stats_kernel<<<grid, CE_THREADS, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)logits, ld, rows, cols, targets, vocab_start,
                                                                ignore_index, row_max, row_sum, target_logit, loss);
  MESH_CUDA_OK(cudaGetLastError());
  return 0;
}

extern "C" int mesh_ce_stats_bf16(const void* logits, long long ld, int rows, int cols, const long long* targets,
                                  long long vocab_start, long long ignore_index, float* row_max, float* row_sum,
                                  float* target_logit, void* stream) {
  return mesh_ce_loss_bf16(logits, ld, rows, cols, targets, vocab_start, ignore_index, row_max, row_sum, target_logit, nullptr, stream);
}

extern "C" int mesh_ce_reduce(const float* loss, const long long* targets, int rows, long long ignore_index, int mean, float* out,
                              float* divisor, void* stream) {
  using namespace mesh;
  if (!out || !divisor || (rows > 0 && (!loss || !targets))) return set_error(-2, "ce_reduce: null argument");
  ce_reduce_kernel<<<1, 1024, 0, (cudaStream_t)stream>>>(loss, targets, rows, ignore_index, mean, out, divisor);
  MESH_CUDA_OK(cudaGetLastError());
  return 0;
}

extern "C" int mesh_ce_grad_of_bf16(const void* logits, long long ld, void* dlogits, long long ldd, int rows, int cols,
                                    const long long* targets, long long vocab_start, long long ignore_index, const float* gmax,
                                    const float* gsum, const float* g, int g_stride, const float* divisor, void* stream) {
  using namespace mesh;
  if (rows <= 0 || cols <= 0) return 0;
  if (!logits || !dlogits || !targets || !gmax || !gsum || !g) return set_error(-2, "ce_grad: null argument");
  int grid = rows < 148 * 8 ? rows : 148 * 8;
  ce_grad_kernel<<<grid, CE_THREADS, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)logits, ld, (__nv_bfloat16*)dlogits, ldd, rows, cols,
                                                               targets, vocab_start, ignore_index, gmax, gsum, g, g_stride, divisor);
  MESH_CUDA_OK(cudaGetLastError());
  return 0;
}

extern "C" int mesh_ce_grad_bf16(const void* logits, long long ld, void* dlogits, long long ldd, int rows, int cols,
                                 const long long* targets, long long vocab_start, const float* gmax, const float* gsum,
                                 const float* gscale, void* stream) {
  constexpr long long none = (long long)(1ull << 63);        // gscale is zero in ignored rows already
  return mesh_ce_grad_of_bf16(logits, ld, dlogits, ldd, rows, cols, targets, vocab_start, none, gmax, gsum, gscale, 1, nullptr, stream);
}
