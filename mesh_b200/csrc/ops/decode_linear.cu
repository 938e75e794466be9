// Stand-alone launches of the decode-time linear layer (the layer itself: decode_linear.cuh).
#include <cuda.h>
#include "decode_linear.cuh"

namespace mesh {
namespace decode {

// A decoder step is a chain of dependent launches of a few microseconds each, so what counts is that HBM does not idle
// between them and that nobody waits for a load he could have asked for earlier.  A ninth warp streams the CTA's weights
// through a ring of stages that fills an SM's shared memory; weights depend on no earlier kernel, so the ring is filled
// before the launch waits for the kernel before it, and the computing warps never wait for more than their stage.  The
// copies are tiles of a tensor map, eight rows by 128 bytes by eight chunks: the same stream as one bulk copy per row and
// stage (1 KB) ran at half the rate.
//
// One decode call of five layers and the head, with the attention and selection kernels of this directory: bf16, batch 1,
// head of 262144 498 -> 366 us; 4-bit, batch 8, head of 65536 419 -> 261 us.  Alone (bf16, batch 1, back to back, before -> now; HBM
// at the measured copy rate): 2048 -> 3072 5.7 -> 4.7 us (1.9), gate and up 2048 -> 2 x 8192 17.0 -> 12.4 us (10.2),
// 8192 -> 2048 11.9 -> 6.7 us (5.1), head 2048 -> 262144 193 -> 151 us (164).  4-bit, batch 8: 7.4 -> 5.4, 16.7 -> 10.3,
// 9.2 -> 7.8, 135 -> 103 us: there a group of 16 rows is one stage, and its barrier and epilogue bound it.
constexpr int STREAM_THREADS = THREADS + 32;
constexpr int MAX_STAGES = 16;
constexpr size_t WHOLE_SMEM = 226 * 1024;           // of 227 KB: the barriers and a few words are static

struct ComputeBar { __device__ __forceinline__ void operator()() const { asm volatile("bar.sync 1, %0;" ::"n"(THREADS) : "memory"); } };

// A stage: KC 128-byte chunks of each of the 16 rows of a group, as [chunk][8 rows][128 B] for the first eight rows and
// again for the others, 128-byte swizzled, then the rows' scales.  Warp w multiplies chunk w (U = 2), or half of chunk
// w / 2 (U = 1) when K is too short for eight chunks.
template <int W4, int U> struct StreamGeom {
  static constexpr int KPC = W4 == 0 ? 64 : W4 == 3 ? 128 : 256;          // k per chunk
  static constexpr int KC = 4 * U;
  static constexpr int KT = KPC * KC;                                     // k per stage
  static constexpr int HALF = KC * 8 * 128;                               // bytes of eight rows
  static constexpr int SROWB = W4 == 0 ? 0 : KT / 32;                     // bytes of one row's scales
  static constexpr int SLOT = 2 * HALF + (W4 == 0 ? 0 : 1024);
  static constexpr int TX = 2 * HALF + 16 * SROWB;
};


__host__ __device__ inline size_t stream_fixed_bytes(int K, int B, int w4) {
  return lin_smem_bytes(K, B) + xsum_bytes(K, w4);
}

struct StreamMaps { CUtensorMap w, s; };      // weights [chunk][row][128 B]; scales [row][K / 64]

template <int W4, int U>
__global__ void __launch_bounds__(STREAM_THREADS) decode_stream_kernel(const LinArgs a, const __grid_constant__ StreamMaps maps,
                                                                         int n_stages) {
  using G = StreamGeom<W4, U>;
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ __align__(8) unsigned long long bars[2 * MAX_STAGES];
  __shared__ int dead_s;
  volatile int* dead = &dead_s;
  const uint32_t full0 = smem_u32(bars), empty0 = full0 + 8 * MAX_STAGES;
  const uint32_t ring = (smem_u32(smem) + (uint32_t)stream_fixed_bytes(a.K, a.B, W4 == 2 ? 1 : 0) + 1023u) & ~1023u;
  const uint8_t* ring_p = smem + (ring - smem_u32(smem));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // Let the next kernel of the stream start its own weight requests now.
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (threadIdx.x == 0) {
    for (int s = 0; s < n_stages; ++s) {
      mbar_init(full0 + 8 * s, 1);
      mbar_init(empty0 + 8 * s, WARPS);
    }
    dead_s = 0;
    fence_mbar_init();
  }
  __syncthreads();
  const int K = a.K, kstages = K / G::KT;
  if (warp == WARPS) {
    // ---------------------------------------------------------------- weights
    if (lane != 0) return;
    int stage = 0, n = 0;
    for (int grp = blockIdx.x; grp < a.n_groups; grp += gridDim.x) {
      int rA, rB;
      group_rows(a, grp, rA, rB);
      for (int ks = 0; ks < kstages; ++ks, ++n) {
        const uint32_t full = full0 + 8 * stage;
        if (n >= n_stages && !mbar_wait(empty0 + 8 * stage, ((n / n_stages) - 1) & 1, dead, a.status, SITE_SMEM_EMPTY)) goto drain;
        mbar_expect_tx(full, G::TX);
        const uint32_t slot = ring + (uint32_t)stage * G::SLOT;
        tma_load_3d(slot, &maps.w, full, 0, rA, ks * G::KC);
        tma_load_3d(slot + G::HALF, &maps.w, full, 0, rB, ks * G::KC);
        if (W4 != 0) {
          tma_load_2d(slot + 2 * G::HALF, &maps.s, full, ks * (G::KT / 64), rA);
          tma_load_2d(slot + 2 * G::HALF + 8 * G::SROWB, &maps.s, full, ks * (G::KT / 64), rB);
        }
        if (++stage == n_stages) stage = 0;
      }
    }
  drain:
    // The CTA's shared memory has to stay until the last copies have landed in it, also when the computing warps gave up on
    // them: nobody else waits then.  (A flag in the loops instead of the jump made the chain of 4-bit layers 5 % slower.)
    const unsigned long long t0 = globaltimer_ns();
    for (int i = max(0, n - n_stages); i < n; ++i)
      while (!mbar_try_wait(full0 + 8 * (i % n_stages), (i / n_stages) & 1) && globaltimer_ns() - t0 < MESH_WAIT_LIMIT_NS) { __nanosleep(100); }
    return;
  }
  // ------------------------------------------------------------------ products
  if (a.norm_w)                                                   // constant too: on its way before the wait
    for (int v = threadIdx.x * 64; v < K; v += THREADS * 64) asm volatile("prefetch.global.L2 [%0];" ::"l"(a.norm_w + v));
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int xstride = K * 2 + a.xpad;
  uint8_t* xs = smem;
  float* red = reinterpret_cast<float*>(smem + (size_t)a.B * (K * 2 + XPAD));
  const int g8 = lane >> 2, t4 = lane & 3;
  // The row of the tile a lane reads.  128-bit reads (bf16, 8-bit): rows whose swizzle differs in bit 2 sit next to each
  // other; 64-bit reads (4-bit): four even rows, then four odd ones.  The lanes of one phase then cover all banks.
  const int row = W4 == 2 ? ((g8 & 3) << 1) | (g8 >> 2) : (g8 >> 1) | ((g8 & 1) << 2);
  constexpr int CH = G::KT / WARPS;                               // k per warp and stage
  const int chunk = U == 2 ? warp : warp >> 1, c0 = U == 2 ? 0 : (warp & 1) * 4;
  stage_x(a, xs, xstride, ComputeBar{});
  prefetch_next(a, THREADS);
  const uint8_t* xrow = xs + (g8 < a.B ? g8 : a.B - 1) * xstride + (warp * CH + t4 * (W4 == 0 ? 8 : 16)) * 2;
  float* xsum = red + 2 * RED_FLOATS;                             // [K / 64][NB], 4-bit codes only
  if constexpr (W4 == 2) sum_x(a, xs, xstride, xsum, ComputeBar{});
  float c[4] = {0.f, 0.f, 0.f, 0.f};
  int stage = 0, turn = 0;
  uint32_t phase = 0;
  for (int grp = blockIdx.x; grp < a.n_groups; grp += gridDim.x, turn ^= 1) {
    for (int ks = 0; ks < kstages; ++ks) {
      // after a wait has run out nobody waits any more (the status block says why the results are garbage), but every
      // thread still meets every barrier; a stage whose copy was not seen to land is not given back
      const bool landed = !*dead && mbar_wait(full0 + 8 * stage, phase, dead, a.status, SITE_SMEM_FULL);
      const uint8_t* slot = ring_p + (uint32_t)stage * G::SLOT;
      const uint8_t* ra = slot + chunk * 1024 + row * 128;
      const uint8_t* xp = xrow + (size_t)ks * G::KT * 2;
      if constexpr (W4 == 0) {
        Chunk<W4, U> ch;
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const uint8_t* w = ra + (((c0 + u * 4 + t4) ^ row) << 4);
          ch.a[u] = at<uint4>(w);
          ch.b[u] = at<uint4>(w + G::HALF);
        }
        mma_chunk<W4, U>(ch, xp, c);
      } else {
        constexpr int GROUPS = CH / 64;
        const uint8_t* sc = slot + 2 * G::HALF + row * G::SROWB + warp * GROUPS * 2;
        const int g0 = (ks * G::KT + warp * CH) / 64;
#pragma unroll
        for (int g = 0; g < GROUPS; ++g) {
          const uint8_t* w = ra + (W4 == 2 ? (((c0 + 2 * g + (t4 >> 1)) ^ row) << 4) + (t4 & 1) * 8 : ((c0 + 4 * g + t4) ^ row) << 4);
          mma_codes<W4>(w, w + G::HALF, __half2float(at<__half>(sc + 2 * g)), __half2float(at<__half>(sc + 8 * G::SROWB + 2 * g)),
                        W4 == 2 ? *reinterpret_cast<const float2*>(xsum + (g0 + g) * NB + 2 * t4) : make_float2(0.f, 0.f), xp + g * 128, c);
        }
      }
      __syncwarp();
      if (lane == 0 && landed) mbar_arrive(empty0 + 8 * stage);
      if (++stage == n_stages) { stage = 0; phase ^= 1u; }
    }
    finish_group(a, grp, c, row, red + turn * RED_FLOATS, ComputeBar{});
    c[0] = c[1] = c[2] = c[3] = 0.f;
  }
}

// Weights read into registers: where no ring fits beside x, and rows and scales that the copies do not take.
template <int W4, int U>
__global__ void __launch_bounds__(THREADS) decode_linear_kernel(const LinArgs a) {
  extern __shared__ __align__(128) uint8_t smem[];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  linear_body<W4, U>(a, smem, [] { asm volatile("griddepcontrol.wait;" ::: "memory"); });
}

template <class... KArgs, class... Args>
static int launch(void (*kern)(KArgs...), int grid, int threads, size_t smem, void* stream, Args... args) {
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = (cudaStream_t)stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = pdl_enabled() ? 1 : 0;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  MESH_CUDA_OK(cudaLaunchKernelEx(&cfg, kern, args...));
  MESH_CUDA_OK(cudaGetLastError());
  return 0;
}

// weights as [128-byte chunk][row][128 B]: a box of `rows` rows and `chunks` chunks arrives as swizzled slabs
static bool weight_map(CUtensorMap* m, const MeshDecodeLinear* d, cuuint64_t rows, cuuint32_t box_rows, cuuint32_t chunks) {
  const cuuint64_t row_bytes = (cuuint64_t)(d->w4 == 0 ? d->K * 2 : d->w4 == 8 ? d->K : d->K / 2);
  const cuuint64_t dims[3] = {128, rows, row_bytes / 128}, strides[2] = {row_bytes, 128};
  const cuuint32_t box[3] = {128, box_rows, chunks}, ones[3] = {1, 1, 1};
  return encode_tiled(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, d->w, dims, strides, box, ones, CU_TENSOR_MAP_SWIZZLE_128B);
}
static long long weight_rows(const MeshDecodeLinear* d, const LinArgs& a) {
  return d->mode == MESH_DEC_GLU && a.up_off > 0 ? (long long)a.up_off + d->N : (long long)d->N;
}

static int grid_of(const LinArgs& a) { return a.n_groups < sm_count() ? a.n_groups : sm_count(); }
template <int W4, int U>
static long long stages_read(const MeshDecodeLinear* d, const LinArgs& a) {
  return (long long)((a.n_groups + grid_of(a) - 1) / grid_of(a)) * (d->K / StreamGeom<W4, U>::KT);
}
// Stages of the ring: all that fit beside x, at most what the CTA reads.  A ring of half an SM's shared memory, which would
// let the next launch fill its own while this one runs, was slower over the whole step (bf16, batch 1, five layers and
// the head, kernel time: 376 us against 341; 4-bit, batch 8: 288 against 249).
template <int W4, int U>
static int ring_stages(const MeshDecodeLinear* d, const LinArgs& a) {
  using G = StreamGeom<W4, U>;
  if (d->K % G::KT) return 0;
  const size_t fixed = stream_fixed_bytes(d->K, d->B, d->w4) + 1024;      // and the alignment of the ring
  long long n = fixed < WHOLE_SMEM ? (long long)((WHOLE_SMEM - fixed) / G::SLOT) : 0;
  if (n > MAX_STAGES) n = MAX_STAGES;
  return (int)(n < stages_read<W4, U>(d, a) ? n : stages_read<W4, U>(d, a));
}

template <int W4, int U>
static int launch_stream(const MeshDecodeLinear* d, const LinArgs& a, void* stream) {
  using G = StreamGeom<W4, U>;
  auto kern = decode_stream_kernel<W4, U>;
  static bool configured = false;
  if (!configured) {
    MESH_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, WHOLE_SMEM));
    configured = true;
  }
  const cuuint64_t rows = (cuuint64_t)weight_rows(d, a);
  StreamMaps maps;
  memset(&maps, 0, sizeof(maps));
  if (!weight_map(&maps.w, d, rows, 8, G::KC)) return last_error_code();
  if constexpr (W4 != 0) {
    const cuuint64_t dims[2] = {(cuuint64_t)(d->K / 64), rows}, strides[1] = {(cuuint64_t)(d->K / 32)};
    const cuuint32_t box[2] = {(cuuint32_t)(G::KT / 64), 8}, ones[2] = {1, 1};
    if (!encode_tiled(&maps.s, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, d->scales, dims, strides, box, ones, CU_TENSOR_MAP_SWIZZLE_NONE))
      return last_error_code();
  }
  const int stages = ring_stages<W4, U>(d, a);
  const size_t fixed = stream_fixed_bytes(d->K, d->B, d->w4) + 1024;
  return launch(kern, grid_of(a), STREAM_THREADS, fixed + stages * G::SLOT, stream, a, maps, stages);
}

template <int W4, int U>
static int launch_registers(const MeshDecodeLinear* d, const LinArgs& a, void* stream) {
  auto kern = decode_linear_kernel<W4, U>;
  static bool configured = false;
  if (!configured) {
    MESH_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)LIN_SMEM_MOST));
    configured = true;
  }
  const size_t smem = lin_smem_bytes(d->K, d->B);
  const int cap = sm_count() * (smem > 100 * 1024 ? 1 : 2);
  return launch(kern, a.n_groups < cap ? a.n_groups : cap, THREADS, smem, stream, a);
}

// The register reader with the widest steps that a warp's slice of K is a multiple of.
static int launch_registers(const MeshDecodeLinear* d, LinArgs a, int variant, void* stream) {
  switch (variant) {
    case LIN_W4W_U2: return launch_registers<2, 2>(d, a, stream);
    case LIN_W4W_U1: a.xpad = XPAD; return launch_registers<1, 2>(d, a, stream);
    case LIN_W4N_U2: return launch_registers<1, 2>(d, a, stream);
    case LIN_W4N_U1: return launch_registers<1, 1>(d, a, stream);
    case LIN_W8_U4: return launch_registers<3, 4>(d, a, stream);
    case LIN_W8_U2: return launch_registers<3, 2>(d, a, stream);
    case LIN_W8_U1: return launch_registers<3, 1>(d, a, stream);
    case LIN_BF16_U4: return launch_registers<0, 4>(d, a, stream);
    default: return launch_registers<0, 1>(d, a, stream);
  }
}

// A ring needs two stages, or copies and products take turns: N = 4096, batch 8, bf16, K = 11776 with two stages 33 us, 12288
// with one 55.  Stages of half the size come next, and registers where those do not fit twice either.  Where the register
// reader's widest step divides a warp's slice it is the better of the two (bf16, K = 12288: 35 us, half stages 41; 8-bit 28
// and 31); its narrow step is not (bf16, K = 12800: 83 and 56), and 4-bit codes would be rounded in its widest one.
template <int W4>
static int launch_reader(const MeshDecodeLinear* d, const LinArgs& a, int variant, void* stream) {
  const int wide = ring_stages<W4, 2>(d, a), half = ring_stages<W4, 1>(d, a);
  const bool quick = variant == LIN_BF16_U4 || variant == LIN_W8_U4;
  if (wide >= 2 || (wide == 1 && stages_read<W4, 2>(d, a) == 1)) return launch_stream<W4, 2>(d, a, stream);
  if ((half >= 2 && !quick) || (half == 1 && stages_read<W4, 1>(d, a) == 1)) return launch_stream<W4, 1>(d, a, stream);
  return launch_registers(d, a, variant, stream);
}

}  // namespace decode
}  // namespace mesh

using namespace mesh;
using namespace mesh::decode;

extern "C" int mesh_decode_linear(const MeshDecodeLinear* d, void* stream) {
  LinArgs a;
  int variant = 0;
  const int rc = lin_prepare(d, a, variant);
  if (rc) return rc;
  // 4-bit rows that are not whole 128-byte chunks, and scales off the 16-byte grid, are not for the copy engine
  if (variant == LIN_W4N_U2 || variant == LIN_W4N_U1 || (d->w4 && (uintptr_t)d->scales % 16)) return launch_registers(d, a, variant, stream);
  return d->w4 == 8 ? launch_reader<3>(d, a, variant, stream) : d->w4 ? launch_reader<2>(d, a, variant, stream)
                                                                      : launch_reader<0>(d, a, variant, stream);
}
