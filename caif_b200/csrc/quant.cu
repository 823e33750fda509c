// Quantize / dequantize / cast kernels.
//
// Results are bit-identical to the reference's kernels in
// src/caif_cuda_kernels_quant.cu (same fp32 operations in the same order per
// element; only the parallel decomposition differs):
//   int8 per-tensor   :384-483    int8 per-channel  :502-620
//   int4 per-group    :205-362    casts             :38-199
// The reference quantizes int4 with one thread per group and serial 128-element
// loops; here a warp owns a group (coalesced float4/float2 loads, shuffle
// max-reduce), which is what makes load-time quantization of a multi-GB model
// bandwidth-bound instead of latency-bound.
#include "common.cuh"

namespace caifq
{

namespace
{

constexpr int kBlock = 256;

__device__ __forceinline__ float warp_max(float v)
{
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
  {
    v = fmaxf(v, __shfl_xor_sync(0xFFFFFFFFu, v, o));
  }
  return v;
}

// |x| maximum that ignores NaN exactly like `if (fabsf(x) > m) m = fabsf(x)`.
__device__ __forceinline__ float absmax_step(float m, float x)
{
  const float a = fabsf(x);
  return (a > m) ? a : m;
}

__device__ __forceinline__ float clamp_sym(float v, float lim)
{
  if (v > lim)
  {
    v = lim;
  }
  else if (v < -lim)
  {
    v = -lim;
  }
  return v;
}

// ---------------------------------------------------------------- int8 / tensor

// Three launches, each placed while the one before it still runs: the blocks' maxima, the scale, the codes.  Small and
// middling tensors are bound by the launches (us, a cleared scale, atomic maxima and plain launches / now: 309 x 768 12.1 / 7.3,
// 2000 x 4096 18.5 / 12.5, 14336 x 4096 84 / 80).  The maxima lie where the codes will: the caller has no scratch.
__device__ __forceinline__ void after_previous_kernel()
{
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

__device__ __forceinline__ float block_max(float m)
{
  __shared__ float part[kBlock / 32];
  m = warp_max(m);
  if ((threadIdx.x & 31) == 0)
  {
    part[threadIdx.x >> 5] = m;
  }
  __syncthreads();
  return warp_max((threadIdx.x & 31) < kBlock / 32 ? part[threadIdx.x & 31] : 0.0f);
}

constexpr int kAbsmaxLoads = 8;   // 16-byte loads in flight per thread

__global__ void __launch_bounds__(kBlock) absmax_kernel(const float *x, uint8_t *maxima, int64_t n)
{
  after_previous_kernel();
  float m = 0.0f;
  if ((reinterpret_cast<uintptr_t>(x) & 15u) == 0)
  {
    const float4 *x4 = reinterpret_cast<const float4 *>(x);
    const int64_t n4 = n >> 2;
    const int64_t step = static_cast<int64_t>(gridDim.x) * kBlock * kAbsmaxLoads;
    for (int64_t base = static_cast<int64_t>(blockIdx.x) * (kBlock * kAbsmaxLoads) + threadIdx.x; base < n4; base += step)
    {
      float4 v[kAbsmaxLoads];
#pragma unroll
      for (int u = 0; u < kAbsmaxLoads; ++u)
      {
        const int64_t j = base + u * kBlock;
        v[u] = j < n4 ? x4[j] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      }
#pragma unroll
      for (int u = 0; u < kAbsmaxLoads; ++u)
      {
        m = absmax_step(absmax_step(absmax_step(absmax_step(m, v[u].x), v[u].y), v[u].z), v[u].w);
      }
    }
    const int64_t rest = (n4 << 2) + threadIdx.x;
    if (blockIdx.x == 0 && rest < n)
    {
      m = absmax_step(m, x[rest]);
    }
  }
  else
  {
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride)
    {
      m = absmax_step(m, x[i]);
    }
  }
  m = block_max(m);
  if (threadIdx.x < 4)
  {
    // (byte by byte: the codes may start anywhere)
    maxima[4 * static_cast<int64_t>(blockIdx.x) + threadIdx.x] =
        static_cast<uint8_t>(__float_as_uint(m) >> (8 * threadIdx.x));
  }
}

__global__ void __launch_bounds__(kBlock) finalize_scale_kernel(const uint8_t *maxima, int count, float *scale)
{
  after_previous_kernel();
  float m = 0.0f;
  for (int i = static_cast<int>(threadIdx.x); i < count; i += kBlock)
  {
    const uint8_t *b = maxima + 4 * i;
    m = fmaxf(m, __uint_as_float(static_cast<uint32_t>(b[0]) | (static_cast<uint32_t>(b[1]) << 8) |
                                 (static_cast<uint32_t>(b[2]) << 16) | (static_cast<uint32_t>(b[3]) << 24)));
  }
  m = block_max(m);
  if (threadIdx.x == 0)
  {
    scale[0] = (m > 0.0f) ? __fdiv_rn(m, 127.0f) : 1.0f;
  }
}

__device__ __forceinline__ int quant_int8(float x, float inv)
{
  return static_cast<int>(rintf(clamp_sym(__fmul_rn(x, inv), 127.0f)));
}

__device__ __forceinline__ uint32_t quant_int8x4(const float4 v, const float4 inv)
{
  return (static_cast<uint32_t>(quant_int8(v.x, inv.x)) & 0xFFu) |
         ((static_cast<uint32_t>(quant_int8(v.y, inv.y)) & 0xFFu) << 8) |
         ((static_cast<uint32_t>(quant_int8(v.z, inv.z)) & 0xFFu) << 16) |
         ((static_cast<uint32_t>(quant_int8(v.w, inv.w)) & 0xFFu) << 24);
}

// Four 16-byte loads in flight a thread, and the blocks take the elements from the end: the maximum's pass has just
// left the last of them in L2.
constexpr int kInt8Loads = 4;

__global__ void __launch_bounds__(kBlock)
quantize_int8_pt_kernel(const float *x, int8_t *q, const float *scale, int64_t n)
{
  after_previous_kernel();
  const float s = scale[0];
  const float inv = (s > 0.0f) ? __fdiv_rn(1.0f, s) : 0.0f;
  const int64_t block = static_cast<int64_t>(gridDim.x) - 1 - blockIdx.x;
  if (((reinterpret_cast<uintptr_t>(x) & 15u) | (reinterpret_cast<uintptr_t>(q) & 3u)) == 0)
  {
    const int64_t n4 = n >> 2;
    const int64_t base = block * (kBlock * kInt8Loads) + threadIdx.x;
    float4 v[kInt8Loads];
#pragma unroll
    for (int u = 0; u < kInt8Loads; ++u)
    {
      const int64_t j = base + u * kBlock;
      v[u] = j < n4 ? __ldcs(reinterpret_cast<const float4 *>(x) + j) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
#pragma unroll
    for (int u = 0; u < kInt8Loads; ++u)
    {
      const int64_t j = base + u * kBlock;
      if (j < n4)
      {
        reinterpret_cast<uint32_t *>(q)[j] = quant_int8x4(v[u], make_float4(inv, inv, inv, inv));
      }
    }
    const int64_t rest = (n4 << 2) + threadIdx.x;
    if (block == 0 && rest < n)
    {
      q[rest] = static_cast<int8_t>(quant_int8(x[rest], inv));
    }
  }
  else
  {
    const int64_t first = block * (kBlock * kInt8Loads * 4);
    const int64_t last = (first + kBlock * kInt8Loads * 4 < n) ? first + kBlock * kInt8Loads * 4 : n;
    for (int64_t j = first + threadIdx.x; j < last; j += kBlock)
    {
      q[j] = static_cast<int8_t>(quant_int8(x[j], inv));
    }
  }
}

__global__ void dequantize_int8_pt_kernel(const int8_t *__restrict__ q, float *__restrict__ out,
                                          const float *__restrict__ scale, int64_t n)
{
  const float s = scale[0];
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride)
  {
    out[i] = __fmul_rn(static_cast<float>(q[i]), s);
  }
}

// --------------------------------------------------------------- int8 / channel

// One launch: a cluster of eight CTAs owns W columns, each CTA a slice of the rows.  The CTAs' column maxima meet through
// distributed shared memory, and each quantizes its slice, from its last rows on: the first pass has just left those in L2.
// A lane takes 16 bytes of a row, W / 4 lanes a row.  Small tensors are bound by the launch, large ones by reading twice.
// (us, clearing the scales, atomic maxima, a launch for the scales and one for the codes / now: 1084 x 2176 13.3 / 6.2, 2000 x
// 4096 18.6 / 11.7, 14336 x 4096 93.7 / 92.0.)
constexpr int kPcSlices = 8;

template <int W, int THREADS>
__global__ void __launch_bounds__(THREADS)
quantize_int8_pc_kernel(const float *x, int8_t *q, float *scales, int rows, int cols, int vec)
{
  constexpr int LANES = W / 4;                          // of a row
  constexpr int TRIP = (THREADS / 32) * (32 / LANES);    // rows the block takes at a time
  __shared__ float part[THREADS / 32][W];
  __shared__ float most[W];
  __shared__ float inv_of[W];
  after_previous_kernel();
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int c0 = static_cast<int>(blockIdx.x) * W;
  const int c = c0 + 4 * (lane % LANES);
  const int per = (rows + kPcSlices - 1) / kPcSlices;
  const int slice = static_cast<int>(blockIdx.y);       // (the cluster is the grid's second dimension)
  const int r_begin = min(rows, slice * per);
  const int r_end = min(rows, r_begin + per);
  const int mine = warp * (32 / LANES) + lane / LANES;
  auto load = [&](int r)
  {
    float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (r >= r_begin && r < r_end)
    {
      const float *row = x + static_cast<int64_t>(r) * cols;
      if (vec)
      {
        if (c < cols)
        {
          v = *reinterpret_cast<const float4 *>(row + c);
        }
      }
      else
      {
        v.x = (c + 0 < cols) ? row[c + 0] : 0.0f;
        v.y = (c + 1 < cols) ? row[c + 1] : 0.0f;
        v.z = (c + 2 < cols) ? row[c + 2] : 0.0f;
        v.w = (c + 3 < cols) ? row[c + 3] : 0.0f;
      }
    }
    return v;
  };
  float m[4] = {0.0f, 0.0f, 0.0f, 0.0f};
  constexpr int U = 8;
  for (int r = r_begin + mine; r - mine < r_end; r += U * TRIP)
  {
    float4 v[U];
#pragma unroll
    for (int u = 0; u < U; ++u)
    {
      v[u] = load(r + u * TRIP);
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
    {
      m[0] = absmax_step(m[0], v[u].x);
      m[1] = absmax_step(m[1], v[u].y);
      m[2] = absmax_step(m[2], v[u].z);
      m[3] = absmax_step(m[3], v[u].w);
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
  {
#pragma unroll
    for (int off = LANES; off < 32; off <<= 1)
    {
      m[i] = fmaxf(m[i], __shfl_xor_sync(0xFFFFFFFFu, m[i], off));
    }
    if (lane < LANES)
    {
      part[warp][4 * lane + i] = m[i];
    }
  }
  __syncthreads();
  if (threadIdx.x < W)
  {
    float best = 0.0f;
#pragma unroll
    for (int w = 0; w < THREADS / 32; ++w)
    {
      best = fmaxf(best, part[w][threadIdx.x]);
    }
    most[threadIdx.x] = best;
  }
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  if (threadIdx.x < W)
  {
    float best = 0.0f;
    const uint32_t local = static_cast<uint32_t>(__cvta_generic_to_shared(&most[threadIdx.x]));
#pragma unroll
    for (int r = 0; r < kPcSlices; ++r)
    {
      uint32_t addr;
      float theirs;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(addr) : "r"(local), "r"(r));
      asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(theirs) : "r"(addr));
      best = fmaxf(best, theirs);
    }
    const float scale = (best > 0.0f) ? __fdiv_rn(best, 127.0f) : 1.0f;
    inv_of[threadIdx.x] = (scale > 0.0f) ? __fdiv_rn(1.0f, scale) : 0.0f;
    if (slice == 0 && c0 + static_cast<int>(threadIdx.x) < cols)
    {
      scales[c0 + threadIdx.x] = scale;
    }
  }
  // (nobody leaves while another CTA may still read its maxima; and inv_of is complete)
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  const int k = 4 * (lane % LANES);
  const float4 inv = make_float4(inv_of[k], inv_of[k + 1], inv_of[k + 2], inv_of[k + 3]);
  constexpr int UQ = 4;
  for (int r = r_end - 1 - mine; r + mine >= r_begin; r -= UQ * TRIP)
  {
    float4 v[UQ];
#pragma unroll
    for (int u = 0; u < UQ; ++u)
    {
      v[u] = load(r - u * TRIP);
    }
#pragma unroll
    for (int u = 0; u < UQ; ++u)
    {
      const int rr = r - u * TRIP;
      if (rr >= r_begin && c < cols)
      {
        int8_t *to = q + static_cast<int64_t>(rr) * cols + c;
        const uint32_t codes = quant_int8x4(v[u], inv);
        if (vec)
        {
          *reinterpret_cast<uint32_t *>(to) = codes;
        }
        else
        {
          for (int i = 0; i < 4 && c + i < cols; ++i)
          {
            to[i] = static_cast<int8_t>(codes >> (8 * i));
          }
        }
      }
    }
  }
}

template <int W, int THREADS>
cudaError_t launch_int8_pc(const float *x, int8_t *q, float *scales, int rows, int cols, int vec, cudaStream_t s)
{
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>((cols + W - 1) / W), kPcSlices);
  cfg.blockDim = dim3(THREADS);
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1;
  attr[0].val.clusterDim.y = kPcSlices;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = dependent_launches() ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, quantize_int8_pc_kernel<W, THREADS>, x, q, scales, rows, cols, vec);
}

// Tall tensors.  Eight slices of the rows leave SMs idle or unevenly loaded there, so the rows are cut as often as fills the
// device.  Column maxima: a block takes 128 columns (a warp one row of them, 16 bytes a lane where rows are aligned) and a
// slice of the rows; its eight warps' maxima meet in shared memory and go to scales[] as an integer atomicMax, which the caller
// cleared.  Then a launch for the scales and one for the codes.  Bound by the launches up to 16384 rows or so (13 to 15 us),
// by reading twice beyond (us, clusters / this: 65536 x 31 42.8 / 23.6, x 256 41 / 30, x 1024 121 / 105; 262144 x 31 160 / 52).
constexpr int kPcCols = 128;

__global__ void __launch_bounds__(kBlock)
channel_absmax_kernel(const float *__restrict__ x, float *__restrict__ scales, int rows, int cols, int rows_per_block,
                      int vec)
{
  __shared__ float part[kBlock / 32][kPcCols];
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int c0 = blockIdx.x * kPcCols;
  const int r_end = min(rows, (static_cast<int>(blockIdx.y) + 1) * rows_per_block);
  float m[4] = {0.0f, 0.0f, 0.0f, 0.0f};
  constexpr int U = 8;
  for (int r = static_cast<int>(blockIdx.y) * rows_per_block + warp; r < r_end; r += U * (kBlock / 32))
  {
    float4 v[U];
#pragma unroll
    for (int u = 0; u < U; ++u)
    {
      const int rr = r + u * (kBlock / 32);
      v[u] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      if (rr < r_end)
      {
        const float *row = x + static_cast<int64_t>(rr) * cols;
        const int c = c0 + 4 * lane;
        if (vec)
        {
          if (c < cols)
          {
            v[u] = *reinterpret_cast<const float4 *>(row + c);
          }
        }
        else
        {
          v[u].x = (c + 0 < cols) ? row[c + 0] : 0.0f;
          v[u].y = (c + 1 < cols) ? row[c + 1] : 0.0f;
          v[u].z = (c + 2 < cols) ? row[c + 2] : 0.0f;
          v[u].w = (c + 3 < cols) ? row[c + 3] : 0.0f;
        }
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
    {
      m[0] = absmax_step(m[0], v[u].x);
      m[1] = absmax_step(m[1], v[u].y);
      m[2] = absmax_step(m[2], v[u].z);
      m[3] = absmax_step(m[3], v[u].w);
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
  {
    part[warp][4 * lane + i] = m[i];
  }
  __syncthreads();
  if (threadIdx.x < kPcCols && c0 + static_cast<int>(threadIdx.x) < cols)
  {
    float best = 0.0f;
#pragma unroll
    for (int w = 0; w < kBlock / 32; ++w)
    {
      best = fmaxf(best, part[w][threadIdx.x]);
    }
    if (best > 0.0f)
    {
      atomicMax(reinterpret_cast<int *>(scales) + c0 + threadIdx.x, __float_as_int(best));
    }
  }
}

__global__ void finalize_channel_scales_kernel(float *scales, int cols)
{
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c < cols)
  {
    const float m = scales[c];
    scales[c] = (m > 0.0f) ? __fdiv_rn(m, 127.0f) : 1.0f;
  }
}

// Same shape of work: a lane keeps its columns' reciprocals and takes the rows of its slice, last slices first (they
// are the ones the maxima's pass left in L2).
__global__ void __launch_bounds__(kBlock)
channel_codes_kernel(const float *__restrict__ x, int8_t *__restrict__ q, const float *__restrict__ scales, int rows,
                        int cols, int rows_per_block, int vec)
{
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int slice = static_cast<int>(gridDim.y) - 1 - static_cast<int>(blockIdx.y);
  const int c = blockIdx.x * kPcCols + 4 * lane;
  const int r_end = min(rows, (slice + 1) * rows_per_block);
  float inv[4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
  {
    const float s = (c + i < cols) ? scales[c + i] : 0.0f;
    inv[i] = (s > 0.0f) ? __fdiv_rn(1.0f, s) : 0.0f;
  }
  constexpr int U = 4;
  for (int r = slice * rows_per_block + warp; r < r_end; r += U * (kBlock / 32))
  {
    if (vec)
    {
      float4 v[U];
#pragma unroll
      for (int u = 0; u < U; ++u)
      {
        const int rr = r + u * (kBlock / 32);
        v[u] = (rr < r_end && c < cols) ? __ldcs(reinterpret_cast<const float4 *>(x + static_cast<int64_t>(rr) * cols + c))
                                        : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      }
#pragma unroll
      for (int u = 0; u < U; ++u)
      {
        const int rr = r + u * (kBlock / 32);
        if (rr < r_end && c < cols)
        {
          *reinterpret_cast<uint32_t *>(q + static_cast<int64_t>(rr) * cols + c) =
              quant_int8x4(v[u], make_float4(inv[0], inv[1], inv[2], inv[3]));
        }
      }
    }
    else
    {
      for (int u = 0; u < U; ++u)
      {
        const int rr = r + u * (kBlock / 32);
        for (int i = 0; i < 4 && rr < r_end && c + i < cols; ++i)
        {
          const int64_t at = static_cast<int64_t>(rr) * cols + c + i;
          q[at] = static_cast<int8_t>(quant_int8(x[at], inv[i]));
        }
      }
    }
  }
}

__global__ void dequantize_int8_pc_kernel(const int8_t *__restrict__ q, float *__restrict__ out,
                                          const float *__restrict__ scales, int64_t total, int cols)
{
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total; i += stride)
  {
    out[i] = __fmul_rn(static_cast<float>(q[i]), scales[i % cols]);
  }
}

// ------------------------------------------------------------------ int4 / group

__device__ __forceinline__ int quant_nibble(float x, float inv)
{
  return static_cast<int>(rintf(clamp_sym(__fmul_rn(x, inv), 7.0f))) & 0xF;
}

// one group, lanes take element pairs (one byte each)
__device__ __forceinline__ void quantize_int4_group(const float *__restrict__ x, uint8_t *__restrict__ packed,
                                                    __half *__restrict__ scales, int64_t n, int group, int64_t g,
                                                    int lane)
{
  const int64_t start = g * group;
  const int64_t end = (start + group < n) ? (start + group) : n;
  float m = 0.0f;
  for (int64_t i = start + 2 * lane; i < end; i += 64)
  {
    m = absmax_step(m, x[i]);
    if (i + 1 < end)
    {
      m = absmax_step(m, x[i + 1]);
    }
  }
  m = warp_max(m);
  const float scale = (m == 0.0f) ? 0.0f : __fdiv_rn(m, 7.0f);
  const float inv = (scale == 0.0f) ? 0.0f : __fdiv_rn(1.0f, scale);
  if (lane == 0)
  {
    scales[g] = __float2half(scale);
  }
  for (int64_t i = start + 2 * lane; i < end; i += 64)
  {
    const int q0 = quant_nibble(x[i], inv);
    const int q1 = (i + 1 < end) ? quant_nibble(x[i + 1], inv) : 0;
    packed[i >> 1] = static_cast<uint8_t>(q0 | (q1 << 4));
  }
}

// Even group size: a warp per group.
__global__ void quantize_int4_warp_kernel(const float *__restrict__ x, uint8_t *__restrict__ packed,
                                          __half *__restrict__ scales, int64_t n, int group, int64_t num_groups)
{
  const int lane = threadIdx.x & 31;
  const int64_t warp = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int64_t warps = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
  for (int64_t g = warp; g < num_groups; g += warps)
  {
    quantize_int4_group(x, packed, scales, n, group, g, lane);
  }
}

// Group sizes 32, 64, 128 and 256 on aligned buffers: a thread keeps eight elements (two 16-byte loads) in registers
// between the maximum and the codes, LPG neighbouring lanes share a group, and kInt4Units such units a thread are
// in flight.  Bound by HBM (4.5 bytes an element); the form above reads every element twice, eight bytes at a time,
// one group in flight a warp (14336 x 4096: 128 us, this one 43).
constexpr int kInt4Units = 4;

template <int LPG>
__global__ void __launch_bounds__(kBlock)
quantize_int4_vec_kernel(const float4 *__restrict__ x, uint32_t *__restrict__ packed, __half *__restrict__ scales,
                         int64_t n, int64_t full_groups)
{
  constexpr int GROUP = LPG * 8;
  const int64_t units = full_groups * LPG;
  const int64_t base = static_cast<int64_t>(blockIdx.x) * (kBlock * kInt4Units) + threadIdx.x;
  float4 v[kInt4Units][2];
#pragma unroll
  for (int u = 0; u < kInt4Units; ++u)
  {
    const int64_t i = base + u * kBlock;
    if (i < units)
    {
      v[u][0] = __ldcs(x + 2 * i);
      v[u][1] = __ldcs(x + 2 * i + 1);
    }
    else
    {
      v[u][0] = v[u][1] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
  }
#pragma unroll
  for (int u = 0; u < kInt4Units; ++u)
  {
    const int64_t i = base + u * kBlock;
    const float e[8] = {v[u][0].x, v[u][0].y, v[u][0].z, v[u][0].w, v[u][1].x, v[u][1].y, v[u][1].z, v[u][1].w};
    float m = 0.0f;
#pragma unroll
    for (int k = 0; k < 8; ++k)
    {
      m = absmax_step(m, e[k]);
    }
#pragma unroll
    for (int o = LPG / 2; o > 0; o >>= 1)
    {
      m = fmaxf(m, __shfl_xor_sync(0xFFFFFFFFu, m, o));
    }
    const float scale = (m == 0.0f) ? 0.0f : __fdiv_rn(m, 7.0f);
    const float inv = (scale == 0.0f) ? 0.0f : __fdiv_rn(1.0f, scale);
    uint32_t w = 0u;
#pragma unroll
    for (int k = 0; k < 8; ++k)
    {
      w |= static_cast<uint32_t>(quant_nibble(e[k], inv)) << (4 * k);
    }
    if (i < units)
    {
      packed[i] = w;
      if ((threadIdx.x & (LPG - 1)) == 0)
      {
        scales[i / LPG] = __float2half(scale);
      }
    }
  }
  // a last, shorter group
  if (blockIdx.x == 0 && threadIdx.x < 32 && full_groups * GROUP < n)
  {
    quantize_int4_group(reinterpret_cast<const float *>(x), reinterpret_cast<uint8_t *>(packed), scales, n, GROUP,
                        full_groups, static_cast<int>(threadIdx.x));
  }
}

template <int LPG>
void launch_int4_vec(const float *x, uint8_t *packed, uint16_t *scales, int64_t n, cudaStream_t s)
{
  const int64_t full = n / (LPG * 8);
  const int64_t per_block = static_cast<int64_t>(kBlock) * kInt4Units;
  const int64_t blocks = (full * LPG + per_block - 1) / per_block;
  quantize_int4_vec_kernel<LPG><<<static_cast<unsigned>(blocks > 0 ? blocks : 1), kBlock, 0, s>>>(
      reinterpret_cast<const float4 *>(x), reinterpret_cast<uint32_t *>(packed), reinterpret_cast<__half *>(scales), n,
      full);
}

// Odd group size: groups share bytes; keep the reference's thread-per-group
// form so the result is whatever the reference's write order yields.
__global__ void quantize_int4_serial_kernel(const float *__restrict__ x, uint8_t *__restrict__ packed,
                                            __half *__restrict__ scales, int64_t n, int group, int64_t num_groups)
{
  const int64_t g = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (g >= num_groups)
  {
    return;
  }
  const int64_t start = g * group;
  const int64_t end = (start + group < n) ? (start + group) : n;
  float m = 0.0f;
  for (int64_t i = start; i < end; ++i)
  {
    m = absmax_step(m, x[i]);
  }
  const float scale = (m == 0.0f) ? 0.0f : __fdiv_rn(m, 7.0f);
  const float inv = (scale == 0.0f) ? 0.0f : __fdiv_rn(1.0f, scale);
  scales[g] = __float2half(scale);
  for (int64_t i = start; i < end; i += 2)
  {
    const int q0 = quant_nibble(x[i], inv);
    const int q1 = (i + 1 < end) ? quant_nibble(x[i + 1], inv) : 0;
    packed[i >> 1] = static_cast<uint8_t>(q0 | (q1 << 4));
  }
}

__global__ void dequantize_int4_kernel(const uint8_t *__restrict__ packed, const __half *__restrict__ scales,
                                       float *__restrict__ out, int64_t n, int group)
{
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  // one byte (two elements) per thread-iteration
  const int64_t nbytes = (n + 1) >> 1;
  for (int64_t b = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; b < nbytes; b += stride)
  {
    const uint8_t v = packed[b];
    const int64_t i0 = b << 1;
    out[i0] = __fmul_rn(static_cast<float>(sign_extend_nibble(v & 0xF)), __half2float(scales[i0 / group]));
    if (i0 + 1 < n)
    {
      out[i0 + 1] = __fmul_rn(static_cast<float>(sign_extend_nibble(v >> 4)), __half2float(scales[(i0 + 1) / group]));
    }
  }
}

// ------------------------------------------------------------------------ casts

template <typename S, typename D>
__device__ __forceinline__ D cast_one(S v);

template <>
__device__ __forceinline__ float cast_one<float, float>(float v) { return v; }
template <>
__device__ __forceinline__ __half cast_one<float, __half>(float v) { return __float2half(v); }
template <>
__device__ __forceinline__ __nv_bfloat16 cast_one<float, __nv_bfloat16>(float v) { return __float2bfloat16(v); }
template <>
__device__ __forceinline__ int8_t cast_one<float, int8_t>(float v)
{
  return static_cast<int8_t>(rintf(clamp_sym(v, 127.0f)));
}
template <>
__device__ __forceinline__ float cast_one<__half, float>(__half v) { return __half2float(v); }
template <>
__device__ __forceinline__ float cast_one<__nv_bfloat16, float>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <>
__device__ __forceinline__ float cast_one<int8_t, float>(int8_t v) { return static_cast<float>(v); }

// Any pair goes through fp32, which is how CAIF_DeviceTensor::To composes them.
template <typename S, typename D>
__global__ void cast_kernel(const S *src, D *dst, int64_t n)
{
  // Launched ahead of the previous kernel's end; the source's address comes out of the wait, so that its read-only loads stay
  // behind it.  Four elements a trip whose loads nothing holds up: neither a bound of their own nor stores that they might
  // overlap (us, bounded and plain / so: 10 M fp32 -> bf16 10.0 / 6.9, 100 M fp32 -> int8 109 / 80; one a trip 8.2 and 90).
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" : "+l"(src)::"memory");
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  for (; i + 3 * stride < n; i += 4 * stride)
  {
    S v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
    {
      v[j] = __ldg(src + i + j * stride);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
    {
      dst[i + j * stride] = cast_one<float, D>(cast_one<S, float>(v[j]));
    }
  }
  for (; i < n; i += stride)
  {
    dst[i] = cast_one<float, D>(cast_one<S, float>(__ldg(src + i)));
  }
}

template <int STORAGE>
__global__ void materialize_kernel(caifq_weight w, void *dst, int dst_dtype, int64_t total)
{
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total; i += stride)
  {
    store_from_float(dst, i, dst_dtype, weight_value<STORAGE>(w, i));
  }
}

inline int grid_for(int64_t n, int per_thread = 1)
{
  const int64_t threads = (n + per_thread - 1) / per_thread;
  int64_t g = (threads + kBlock - 1) / kBlock;
  const int64_t cap = 148 * 16;
  if (g > cap)
  {
    g = cap;
  }
  if (g < 1)
  {
    g = 1;
  }
  return static_cast<int>(g);
}

template <typename S>
int cast_from(const S *src, void *dst, int dst_dtype, int64_t n, cudaStream_t s)
{
  const int g = grid_for(n);
  switch (dst_dtype)
  {
    case CAIFQ_F32:
      CAIFQ_CHECK_CUDA(launch_dependent(cast_kernel<S, float>, dim3(g), dim3(kBlock), 0, s, src, static_cast<float *>(dst), n));
      break;
    case CAIFQ_F16:
      CAIFQ_CHECK_CUDA(launch_dependent(cast_kernel<S, __half>, dim3(g), dim3(kBlock), 0, s, src, static_cast<__half *>(dst), n));
      break;
    case CAIFQ_BF16:
      CAIFQ_CHECK_CUDA(launch_dependent(cast_kernel<S, __nv_bfloat16>, dim3(g), dim3(kBlock), 0, s, src, static_cast<__nv_bfloat16 *>(dst), n));
      break;
    case CAIFQ_I8:
      CAIFQ_CHECK_CUDA(launch_dependent(cast_kernel<S, int8_t>, dim3(g), dim3(kBlock), 0, s, src, static_cast<int8_t *>(dst), n));
      break;
    default:
      set_error("caifq_cast: unsupported destination dtype %d", dst_dtype);
      return CAIFQ_ERR_INVALID;
  }
  CAIFQ_CHECK_LAUNCH();
  return CAIFQ_OK;
}

}  // namespace

int launch_quantize_int8_per_tensor(const float *x, int8_t *q, float *scale, int64_t n, cudaStream_t s)
{
  if (n <= 0)
  {
    return CAIFQ_OK;
  }
  // a block's maximum takes the place of four codes: tensors of fewer have one block, and its bytes go as far as they fit
  const int blocks = grid_for(n, 4 * kAbsmaxLoads);
  uint8_t *maxima = reinterpret_cast<uint8_t *>(q);
  if (n < 4 * static_cast<int64_t>(blocks))
  {
    maxima = reinterpret_cast<uint8_t *>(scale);   // (one block: the scale's own four bytes)
  }
  CAIFQ_CHECK_CUDA(launch_dependent(absmax_kernel, dim3(static_cast<unsigned>(blocks)), dim3(kBlock), 0, s, x, maxima, n));
  CAIFQ_CHECK_CUDA(launch_dependent(finalize_scale_kernel, dim3(1), dim3(kBlock), 0, s, maxima, blocks, scale));
  const int64_t per_block = static_cast<int64_t>(kBlock) * kInt8Loads * 4;
  const int64_t grid = (n + per_block - 1) / per_block;
  CAIFQ_CHECK_CUDA(launch_dependent(quantize_int8_pt_kernel, dim3(static_cast<unsigned>(grid)), dim3(kBlock), 0, s, x, q, scale, n));
  return CAIFQ_OK;
}

int launch_dequantize_int8_per_tensor(const int8_t *q, float *out, const float *scale, int64_t n, cudaStream_t s)
{
  if (n <= 0)
  {
    return CAIFQ_OK;
  }
  dequantize_int8_pt_kernel<<<grid_for(n), kBlock, 0, s>>>(q, out, scale, n);
  CAIFQ_CHECK_LAUNCH();
  return CAIFQ_OK;
}

int launch_quantize_int8_per_channel(const float *x, int8_t *q, float *scales, int rows, int cols, cudaStream_t s)
{
  if (rows <= 0 || cols <= 0)
  {
    return CAIFQ_OK;
  }
  const int vec = (cols % 4) == 0 && (reinterpret_cast<uintptr_t>(x) & 15u) == 0 && (reinterpret_cast<uintptr_t>(q) & 3u) == 0;
  auto ctas = [&](int width) { return (cols + width - 1) / width * kPcSlices; };
  const int sms = device_sm_count();
  // A cluster's CTA walks an eighth of the rows, 2 to 2.5 ns a row (columns that 16-byte loads cannot read 2 to 5); the tall form
  // has its launches, 13 to 17 us, and then the whole device's rate.  So the line lies at a number of rows, lower where rows take
  // longer and where the columns make two to three CTAs of 256 threads an SM, too few loads in flight (us, clusters / tall):
  //   16384 x 31 13.2 / 15.4, x 256 12.4 / 17.4, x 768 23.6 / 24.6, x 2048 50 / 57; 32768 x 128 18.7 / 17.4, x 1536 89 / 85
  //   10240 x 1280 25.0 / 27.2, x 1536 26.5 / 29.8; 14336 x 1280 37.5 / 29.9, x 1536 39.6 / 36.6
  //   off 16 bytes: 4096 x 101 10.7 / 14.4, x 255 11.0 / 17.4; 8192 x 101 17.6 / 14.4; 2048 x 767 14.3 / 16.4, x 1535 13.6 / 19.5;
  //   4096 x 767 22.8 / 18.4, x 1279 24.3 / 21.7, but 8192 x 4095 76 / 90
  const bool few_loads = ctas(32) >= 2 * sms - kPcSlices && ctas(32) < 3 * sms;
  int cluster_rows = few_loads ? 10240 : 16384;
  if (vec == 0 && cols < 3072)
  {
    cluster_rows = cols <= 256 ? 4096 : 2048;
  }
  if (rows > cluster_rows)
  {
    CAIFQ_CHECK_CUDA(cudaMemsetAsync(scales, 0, static_cast<size_t>(cols) * sizeof(float), s));
    const int col_blocks = (cols + kPcCols - 1) / kPcCols;
    // about eight blocks per SM over all columns, at least one trip of eight rows a warp each
    int slices = (sms * 8 + col_blocks - 1) / col_blocks;
    const int most = static_cast<int>((static_cast<int64_t>(rows) + 63) / 64);
    slices = slices < most ? slices : most;
    const int per = static_cast<int>((static_cast<int64_t>(rows) + slices - 1) / slices);
    const dim3 grid(static_cast<unsigned>(col_blocks), static_cast<unsigned>((static_cast<int64_t>(rows) + per - 1) / per));
    channel_absmax_kernel<<<grid, kBlock, 0, s>>>(x, scales, rows, cols, per, vec);
    CAIFQ_CHECK_LAUNCH();
    finalize_channel_scales_kernel<<<(cols + kBlock - 1) / kBlock, kBlock, 0, s>>>(scales, cols);
    CAIFQ_CHECK_LAUNCH();
    channel_codes_kernel<<<grid, kBlock, 0, s>>>(x, q, scales, rows, cols, per, vec);
    CAIFQ_CHECK_LAUNCH();
    return CAIFQ_OK;
  }
  // The widest columns that still give every SM two CTAs; where even 32 of them do not, and there are many rows, 16 and twice
  // the threads (14336 x 512: 27.6 us without), as long as all of its clusters run at a time
  auto launch = launch_int8_pc<32, kBlock>;
  if (ctas(64) >= 2 * sms)
  {
    launch = ctas(128) >= 2 * sms ? launch_int8_pc<128, kBlock> : launch_int8_pc<64, kBlock>;
  }
  else if (ctas(32) < 2 * sms - kPcSlices && rows > 1024)
  {
    launch = launch_int8_pc<16, 2 * kBlock>;
  }
  CAIFQ_CHECK_CUDA(launch(x, q, scales, rows, cols, vec, s));
  return CAIFQ_OK;
}

int launch_dequantize_int8_per_channel(const int8_t *q, float *out, const float *scales, int rows, int cols,
                                       cudaStream_t s)
{
  if (rows <= 0 || cols <= 0)
  {
    return CAIFQ_OK;
  }
  const int64_t total = static_cast<int64_t>(rows) * cols;
  dequantize_int8_pc_kernel<<<grid_for(total), kBlock, 0, s>>>(q, out, scales, total, cols);
  CAIFQ_CHECK_LAUNCH();
  return CAIFQ_OK;
}

int launch_quantize_int4(const float *x, uint8_t *packed, uint16_t *scales, int64_t n, int group, cudaStream_t s)
{
  if (n <= 0)
  {
    return CAIFQ_OK;
  }
  const int64_t num_groups = (n + group - 1) / group;
  const bool aligned = (reinterpret_cast<uintptr_t>(x) & 15u) == 0 && (reinterpret_cast<uintptr_t>(packed) & 3u) == 0;
  if (aligned && group == 128)
  {
    launch_int4_vec<16>(x, packed, scales, n, s);
  }
  else if (aligned && group == 64)
  {
    launch_int4_vec<8>(x, packed, scales, n, s);
  }
  else if (aligned && group == 32)
  {
    launch_int4_vec<4>(x, packed, scales, n, s);
  }
  else if (aligned && group == 256)
  {
    launch_int4_vec<32>(x, packed, scales, n, s);
  }
  else if ((group & 1) == 0)
  {
    const int64_t blocks = (num_groups + (kBlock / 32) - 1) / (kBlock / 32);
    const int64_t cap = 148 * 32;
    quantize_int4_warp_kernel<<<static_cast<unsigned>(blocks < cap ? blocks : cap), kBlock, 0, s>>>(
        x, packed, reinterpret_cast<__half *>(scales), n, group, num_groups);
  }
  else
  {
    quantize_int4_serial_kernel<<<static_cast<unsigned>((num_groups + kBlock - 1) / kBlock), kBlock, 0, s>>>(
        x, packed, reinterpret_cast<__half *>(scales), n, group, num_groups);
  }
  CAIFQ_CHECK_LAUNCH();
  return CAIFQ_OK;
}

int launch_dequantize_int4(const uint8_t *packed, const uint16_t *scales, float *out, int64_t n, int group,
                           cudaStream_t s)
{
  if (n <= 0)
  {
    return CAIFQ_OK;
  }
  dequantize_int4_kernel<<<grid_for((n + 1) / 2), kBlock, 0, s>>>(packed, reinterpret_cast<const __half *>(scales),
                                                                  out, n, group);
  CAIFQ_CHECK_LAUNCH();
  return CAIFQ_OK;
}

int launch_cast(const void *src, int src_dtype, void *dst, int dst_dtype, int64_t n, cudaStream_t s)
{
  if (n <= 0)
  {
    return CAIFQ_OK;
  }
  switch (src_dtype)
  {
    case CAIFQ_F32:
      return cast_from(static_cast<const float *>(src), dst, dst_dtype, n, s);
    case CAIFQ_F16:
      return cast_from(static_cast<const __half *>(src), dst, dst_dtype, n, s);
    case CAIFQ_BF16:
      return cast_from(static_cast<const __nv_bfloat16 *>(src), dst, dst_dtype, n, s);
    case CAIFQ_I8:
      return cast_from(static_cast<const int8_t *>(src), dst, dst_dtype, n, s);
    default:
      set_error("caifq_cast: unsupported source dtype %d", src_dtype);
      return CAIFQ_ERR_INVALID;
  }
}

// ---- codes -> bf16 operand matrix (many-token calls expand the weight once per call / step) ----
// int8: exact bf16 integers with byte permutes and one bf16 subtraction per pair, or the scaled value.  int4: the
// offset-binary nibble is dropped into the mantissa of 2^23 (exact), 2^23 + 8 subtracted (exact), the product with the
// group's fp16 scale rounded once in fp32 and once to bf16 -- the value the reference's dequantize kernel followed by
// its cast to bf16 gives (src/caif_cuda_kernels_quant.cu:364-420, src/caif_device_frozen_linear.cpp:319-334).
// Bound by HBM (2.5 to 3 bytes a weight, most of them writes): 32-byte stores and a shift instead of a 64-bit division
// per unit (64 experts of 2048 x 1408 int4: 101 us a projection before, 84 now).
// blockIdx.y selects the matrix of a run; `units` = weights / 8.
constexpr int kExpandRun = 64;
struct ExpandTable
{
  const void *codes[kExpandRun];
  const void *scales[kExpandRun];
  uint4 *dst[kExpandRun];
  int64_t units[kExpandRun];
};

template <int MODE>
__global__ void expand_kernel(const __grid_constant__ ExpandTable t, GroupOf group_of)
{
  const int e = blockIdx.y;
  const void *codes = t.codes[e];
  const void *scales = t.scales[e];
  // (the scratch may still be read by the kernel before this one; what follows may read the codes and scratch of others.
  // The codes' and scales' addresses come out of the wait, so that their invariant loads stay behind it: a quantizer may be
  // the kernel before)
  asm volatile("griddepcontrol.wait;" : "+l"(codes), "+l"(scales)::"memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  expand_span<MODE>(codes, scales, t.dst[e], t.units[e], group_of);
}

namespace
{
template <int MODE>
int launch_expand(const caifq_weight *ws, int count, uint8_t *dst, cudaStream_t s)
{
  for (int first = 0; first < count; first += kExpandRun)
  {
    const int n = (count - first < kExpandRun) ? (count - first) : kExpandRun;
    ExpandTable t{};
    int64_t most = 0;
    for (int e = 0; e < n; ++e)
    {
      const caifq_weight &w = ws[first + e];
      const int64_t total = static_cast<int64_t>(w.in_dim) * w.out_dim;
      const bool bad_group = MODE == EXPAND_I4 && (w.scales == nullptr || w.group_size <= 0 || (w.group_size % 8) != 0 ||
                                                   w.group_size != ws[0].group_size);
      if ((total % 8) != 0 || bad_group || (MODE == EXPAND_I8_SCALED && w.scales == nullptr) ||
          (reinterpret_cast<uintptr_t>(w.codes) & (MODE == EXPAND_I4 ? 7u : 15u)) != 0 ||
          (reinterpret_cast<uintptr_t>(dst) & 31u) != 0)
      {
        set_error("expand_to_bf16: unsupported weight %d (storage %d)", first + e, w.storage);
        return CAIFQ_ERR_UNSUPPORTED;
      }
      t.codes[e] = w.codes;
      t.scales[e] = w.scales;
      t.dst[e] = reinterpret_cast<uint4 *>(dst);
      t.units[e] = total / 8;
      most = t.units[e] > most ? t.units[e] : most;
      dst += total * 2;
    }
    int gx = grid_for(most, 2);
    const int cap = (148 * 8 + n - 1) / n;   // about eight CTAs per SM over all matrices
    if (gx > cap)
    {
      gx = cap;
    }
    const dim3 grid(static_cast<unsigned>(gx), static_cast<unsigned>(n));
    CAIFQ_CHECK_CUDA(launch_dependent(expand_kernel<MODE>, grid, dim3(kBlock), 0, s, t,
                                      GroupOf::make(MODE == EXPAND_I4 ? ws[0].group_size : 1)));
  }
  return CAIFQ_OK;
}
}  // namespace

int launch_expand_grouped_to_bf16(const caifq_weight *ws, int count, void *dst, cudaStream_t s)
{
  return ws[0].storage == CAIFQ_I8 ? launch_expand<EXPAND_I8>(ws, count, static_cast<uint8_t *>(dst), s)
                                   : launch_expand<EXPAND_I4>(ws, count, static_cast<uint8_t *>(dst), s);
}

// ---- weights as the bf16 matrix the reference's ConvertToComputeDtype would hold for bf16 compute ----
// (src/caif_device_frozen_linear.cpp:288-378): int8 per-tensor bf16(float(code) * scale), int4 as
// expand_int4x8, bf16 copied, fp32 / fp16 rounded to bf16.  Used where several layers' weights are laid one
// under the other into one operand (fused q/k/v), so the scale has to be inside the values.  Neighbours of one
// storage share a launch.
int launch_weights_to_bf16_scaled(const caifq_weight *ws, int count, void *dst, cudaStream_t s)
{
  uint8_t *out = static_cast<uint8_t *>(dst);
  for (int i = 0; i < count;)
  {
    int n = 1;
    while (i + n < count && ws[i + n].storage == ws[i].storage && ws[i + n].group_size == ws[i].group_size)
    {
      ++n;
    }
    int rc = CAIFQ_OK;
    bool aligned = true;
    for (int k = i; k < i + n; ++k)
    {
      const caifq_weight &w = ws[k];
      if ((w.storage == CAIFQ_I8 && (w.scheme != CAIFQ_PER_TENSOR || w.scales == nullptr)) ||
          (w.storage == CAIFQ_I4 && (w.scales == nullptr || w.group_size <= 0 || (w.group_size % 8) != 0)))
      {
        set_error("weight_to_bf16: int8 needs one per-tensor scale, int4 groups of a multiple of 8");
        return CAIFQ_ERR_UNSUPPORTED;
      }
      aligned = aligned && (reinterpret_cast<uintptr_t>(w.codes) & 15u) == 0;
    }
    if (!aligned)
    {
      n = 1;   // a view of codes that 16-byte loads cannot read
      rc = launch_weight_materialize(ws[i], out, CAIFQ_BF16, s);
    }
    else if (ws[i].storage == CAIFQ_I4)
    {
      rc = launch_expand<EXPAND_I4>(ws + i, n, out, s);
    }
    else if (ws[i].storage == CAIFQ_I8)
    {
      rc = launch_expand<EXPAND_I8_SCALED>(ws + i, n, out, s);
    }
    else
    {
      n = 1;
      const int64_t total = static_cast<int64_t>(ws[i].in_dim) * ws[i].out_dim;
      if (ws[i].storage == CAIFQ_BF16)
      {
        CAIFQ_CHECK_CUDA(cudaMemcpyAsync(out, ws[i].codes, static_cast<size_t>(total) * 2, cudaMemcpyDeviceToDevice, s));
      }
      else
      {
        rc = launch_cast(ws[i].codes, ws[i].storage, out, CAIFQ_BF16, total, s);
      }
    }
    if (rc != CAIFQ_OK)
    {
      return rc;
    }
    for (int k = i; k < i + n; ++k)
    {
      out += static_cast<size_t>(ws[k].in_dim) * static_cast<size_t>(ws[k].out_dim) * 2;
    }
    i += n;
  }
  return CAIFQ_OK;
}

int launch_weight_materialize(const caifq_weight &w, void *dst, int dst_dtype, cudaStream_t s)
{
  const int64_t total = static_cast<int64_t>(w.in_dim) * w.out_dim;
  if (total <= 0)
  {
    return CAIFQ_OK;
  }
  const int g = grid_for(total);
  switch (w.storage)
  {
    case CAIFQ_F32:
      materialize_kernel<CAIFQ_F32><<<g, kBlock, 0, s>>>(w, dst, dst_dtype, total);
      break;
    case CAIFQ_F16:
      materialize_kernel<CAIFQ_F16><<<g, kBlock, 0, s>>>(w, dst, dst_dtype, total);
      break;
    case CAIFQ_BF16:
      materialize_kernel<CAIFQ_BF16><<<g, kBlock, 0, s>>>(w, dst, dst_dtype, total);
      break;
    case CAIFQ_I8:
      materialize_kernel<CAIFQ_I8><<<g, kBlock, 0, s>>>(w, dst, dst_dtype, total);
      break;
    case CAIFQ_I4:
      materialize_kernel<CAIFQ_I4><<<g, kBlock, 0, s>>>(w, dst, dst_dtype, total);
      break;
    default:
      set_error("weight_materialize: unsupported storage dtype %d", w.storage);
      return CAIFQ_ERR_INVALID;
  }
  CAIFQ_CHECK_LAUNCH();
  return CAIFQ_OK;
}

}  // namespace caifq
