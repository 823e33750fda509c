// RMSNorm in front of the frozen projections: CAIF_DevicePreNormBlock normalizes, hands the rows to the
// frozen linear (src/caif_device_pre_norm_block.cpp:97-135) and adds the residual.  The reference's kernels
// (src/caif_cuda_kernels_normalization.cu:46-119 forward, :129-203 backward) run one 256-thread block per row,
// thread t owning columns t, t + 256, ..., and read the row twice from global memory with 2- or 4-byte loads.
//
// Here a row comes in once, with 4- to 16-byte loads, into the registers of the warps that own it, both passes read it
// there, and the backward pass keeps its share of grad_gamma in registers over all its rows (the reference issues one
// atomic per element).  A lane plays V adjacent threads of the reference's block.  The kernels with one thread per
// reference thread take the rest (odd row lengths, unaligned rows, rows too long for the registers).  The arithmetic
// of y, rms and dx is the reference's, operation for operation: the same columns per thread in the same order with a
// fused multiply-add per step, the same shuffle-down tree inside a warp, the eight warp sums folded by the same tree,
// IEEE sqrt and divisions -- so those three come out bit-identical.  grad_gamma is a sum over rows whose order the
// reference leaves to its atomics; it agrees to rounding.
#include "common.cuh"

namespace caifq
{

namespace
{

constexpr int kNormThreads = 256;
constexpr int kNormWarps = kNormThreads / 32;
constexpr int kNormMaxPerThread = 32;   // columns a thread can keep of grad_gamma: dim <= 8192

template <typename T>
__device__ __forceinline__ float nf(T v);
template <>
__device__ __forceinline__ float nf<float>(float v) { return v; }
template <>
__device__ __forceinline__ float nf<__half>(__half v) { return __half2float(v); }
template <>
__device__ __forceinline__ float nf<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

template <typename T>
__device__ __forceinline__ T nt(float v);
template <>
__device__ __forceinline__ float nt<float>(float v) { return v; }
template <>
__device__ __forceinline__ __half nt<__half>(float v) { return __float2half(v); }
template <>
__device__ __forceinline__ __nv_bfloat16 nt<__nv_bfloat16>(float v) { return __float2bfloat16(v); }

// sum over the CTA in the reference's order: shuffle-down tree per warp, then the warp sums in lanes 0..7 of
// warp 0 through the same tree; every thread gets the result
__device__ __forceinline__ float block_sum(float v, float *warp_sums)
{
#pragma unroll
  for (int off = 16; off > 0; off >>= 1)
  {
    v += __shfl_down_sync(0xFFFFFFFFu, v, off);
  }
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  __syncthreads();   // the slot array may still be read from the row before
  if (lane == 0)
  {
    warp_sums[warp] = v;
  }
  __syncthreads();
  if (warp == 0)
  {
    v = lane < kNormWarps ? warp_sums[lane] : 0.0f;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
    {
      v += __shfl_down_sync(0xFFFFFFFFu, v, off);
    }
    if (lane == 0)
    {
      warp_sums[kNormWarps] = v;
    }
  }
  __syncthreads();
  return warp_sums[kNormWarps];
}

// row [dim] of T between global and shared memory with 16-byte accesses when `vec`, else element by element
template <int THREADS, typename T>
__device__ __forceinline__ void row_in(T *dst, const T *src, int dim, bool vec)
{
  if (vec)
  {
    const int n16 = dim * static_cast<int>(sizeof(T)) / 16;
    for (int i = threadIdx.x; i < n16; i += THREADS)
    {
      reinterpret_cast<uint4 *>(dst)[i] = __ldg(reinterpret_cast<const uint4 *>(src) + i);
    }
  }
  else
  {
    for (int i = threadIdx.x; i < dim; i += THREADS)
    {
      dst[i] = src[i];
    }
  }
}

template <int THREADS, typename T>
__device__ __forceinline__ void row_out(T *dst, const T *src, int dim, bool vec)
{
  if (vec)
  {
    const int n16 = dim * static_cast<int>(sizeof(T)) / 16;
    for (int i = threadIdx.x; i < n16; i += THREADS)
    {
      reinterpret_cast<uint4 *>(dst)[i] = reinterpret_cast<const uint4 *>(src)[i];
    }
  }
  else
  {
    for (int i = threadIdx.x; i < dim; i += THREADS)
    {
      dst[i] = src[i];
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(kNormThreads, 8)
rmsnorm_fwd_kernel(const T *__restrict__ input, const float *__restrict__ gamma, T *__restrict__ output,
                   float *__restrict__ rms_cache, float epsilon, int rows, int dim, int vec)
{
  extern __shared__ __align__(16) unsigned char norm_smem[];
  __shared__ float warp_sums[kNormWarps + 1];
  T *row = reinterpret_cast<T *>(norm_smem);
  for (int r = blockIdx.x; r < rows; r += gridDim.x)
  {
    __syncthreads();   // the row buffer is free again
    row_in<kNormThreads>(row, input + static_cast<int64_t>(r) * dim, dim, vec != 0);
    __syncthreads();
    float local = 0.0f;
    for (int c = threadIdx.x; c < dim; c += kNormThreads)
    {
      const float v = nf<T>(row[c]);
      local = __fmaf_rn(v, v, local);
    }
    const float total = block_sum(local, warp_sums);
    const float rms = __fsqrt_rn(__fadd_rn(__fdiv_rn(total, static_cast<float>(dim)), epsilon));
    if (threadIdx.x == 0 && rms_cache != nullptr)
    {
      rms_cache[r] = rms;
    }
    const float rstd = __fdiv_rn(1.0f, rms);
    for (int c = threadIdx.x; c < dim; c += kNormThreads)
    {
      row[c] = nt<T>(__fmul_rn(__fmul_rn(nf<T>(row[c]), rstd), __ldg(gamma + c)));
    }
    __syncthreads();
    row_out<kNormThreads>(output + static_cast<int64_t>(r) * dim, row, dim, vec != 0);
  }
}

// ---- rows in registers: a lane plays V adjacent threads of the reference's block ----
// A row is owned by 8 / V warps.  Lane q of virtual threads V q .. V q + V - 1 holds V adjacent columns of every stripe
// of 256, so one access serves them; each of its V partial sums runs over the same columns in the same order as the
// reference's thread.  The shuffle-down tree over 32 virtual threads becomes lane offsets 16 / V ... 1 and then the
// same halving over the lane's own V sums, which adds the same pairs in the same order.
// Bound by HBM for many rows (16-byte loads, one warp a row for 16-bit types, no barrier: 4096 x 4096 bf16 16 us a call, 20 before),
// by latency for few (V = 2: four warps a row, all of it in flight at once).
template <typename T, int V>
struct alignas(V * sizeof(T) < 16 ? V * sizeof(T) : 16) Piece
{
  static constexpr int WORDS = V * static_cast<int>(sizeof(T)) / 4;
  uint32_t w[WORDS];

  __device__ __forceinline__ float get(int i) const
  {
    if constexpr (sizeof(T) == 4)
    {
      return __uint_as_float(w[i]);
    }
    else
    {
      const uint16_t h = static_cast<uint16_t>((i & 1) ? w[i >> 1] >> 16 : w[i >> 1]);
      return nf<T>(*reinterpret_cast<const T *>(&h));
    }
  }

  __device__ __forceinline__ void set(const float (&v)[V])
  {
#pragma unroll
    for (int i = 0; i < WORDS; ++i)
    {
      if constexpr (sizeof(T) == 4)
      {
        w[i] = __float_as_uint(v[i]);
      }
      else
      {
        const T lo = nt<T>(v[2 * i]);
        const T hi = nt<T>(v[2 * i + 1]);
        w[i] = static_cast<uint32_t>(*reinterpret_cast<const uint16_t *>(&lo)) |
               (static_cast<uint32_t>(*reinterpret_cast<const uint16_t *>(&hi)) << 16);
      }
    }
  }

  // the row stays packed between its two passes (the compiler would otherwise keep it as floats: twice the registers)
  __device__ __forceinline__ void keep_packed()
  {
#pragma unroll
    for (int i = 0; i < WORDS; ++i)
    {
      asm volatile("" : "+r"(w[i]));
    }
  }
};

template <typename T, int V>
__device__ __forceinline__ Piece<T, V> zero_piece()
{
  Piece<T, V> p;
#pragma unroll
  for (int i = 0; i < Piece<T, V>::WORDS; ++i)
  {
    p.w[i] = 0u;
  }
  return p;
}

template <int V>
struct Gammas
{
  float e[V];
};

template <int V>
__device__ __forceinline__ Gammas<V> load_gamma(const float *gamma, int c)
{
  Gammas<V> g;
  if constexpr (V == 2)
  {
    const float2 v = __ldg(reinterpret_cast<const float2 *>(gamma + c));
    g.e[0] = v.x;
    g.e[1] = v.y;
  }
  else
  {
#pragma unroll
    for (int i = 0; i < V; i += 4)
    {
      const float4 v = __ldg(reinterpret_cast<const float4 *>(gamma + c + i));
      g.e[i] = v.x;
      g.e[i + 1] = v.y;
      g.e[i + 2] = v.z;
      g.e[i + 3] = v.w;
    }
  }
  return g;
}

// the reference's block sum of its 256 partial sums; every thread of the row gets it.  slots: [8] of this row.
template <int V>
__device__ __forceinline__ float row_sum(float (&v)[V], float *slots, int warp_in_row)
{
  constexpr int LANES = 32 / V;   // lanes of one virtual warp
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int off = LANES / 2; off > 0; off >>= 1)
  {
#pragma unroll
    for (int i = 0; i < V; ++i)
    {
      v[i] += __shfl_down_sync(0xFFFFFFFFu, v[i], off, LANES);
    }
  }
#pragma unroll
  for (int off = V / 2; off > 0; off >>= 1)
  {
#pragma unroll
    for (int i = 0; i < off; ++i)
    {
      v[i] += v[i + off];
    }
  }
  float w[8];
  if constexpr (V == 8)
  {
#pragma unroll
    for (int i = 0; i < 8; ++i)
    {
      w[i] = __shfl_sync(0xFFFFFFFFu, v[0], i * LANES);
    }
  }
  else
  {
    __syncthreads();   // the slots may still be read from the row before
    if ((lane & (LANES - 1)) == 0)
    {
      slots[warp_in_row * V + lane / LANES] = v[0];
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 8; ++i)
    {
      w[i] = slots[i];
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i)
  {
    w[i] += 0.0f;   // lanes 8 to 31 of the reference's last tree
  }
  return ((w[0] + w[4]) + (w[2] + w[6])) + ((w[1] + w[5]) + (w[3] + w[7]));
}

// STRIPES: upper bound of ceil(dim / 256)
template <typename T, int V, int STRIPES>
__global__ void __launch_bounds__(kNormThreads)
rmsnorm_fwd_rows_kernel(const T *input, const float *__restrict__ gamma, T *output,
                        float *__restrict__ rms_cache, float epsilon, int rows, int dim)
{
  constexpr int WARPS = 8 / V;   // per row; V rows per CTA
  __shared__ float sums[V][8];
  // (launched ahead of the previous kernel's end; the next kernel may follow once that one is complete.  gamma's address
  // comes out of the wait, so that its invariant loads stay behind it)
  asm volatile("griddepcontrol.wait;" : "+l"(gamma)::"memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int slot = (threadIdx.x >> 5) / WARPS;
  const int warp_in_row = (threadIdx.x >> 5) % WARPS;
  const int r = blockIdx.x * V + slot;
  const bool live = r < rows;
  const int c0 = (warp_in_row * 32 + (threadIdx.x & 31)) * V;
  const T *src = input + static_cast<int64_t>(live ? r : 0) * dim;
  Piece<T, V> x[STRIPES];
#pragma unroll
  for (int j = 0; j < STRIPES; ++j)
  {
    const int c = c0 + 256 * j;
    x[j] = (live && c < dim) ? *reinterpret_cast<const Piece<T, V> *>(src + c) : zero_piece<T, V>();
  }
  float part[V];
#pragma unroll
  for (int i = 0; i < V; ++i)
  {
    part[i] = 0.0f;
  }
#pragma unroll
  for (int j = 0; j < STRIPES; ++j)
  {
#pragma unroll
    for (int i = 0; i < V; ++i)
    {
      const float v = x[j].get(i);
      part[i] = __fmaf_rn(v, v, part[i]);   // (columns past the row add +0 to a non-negative sum)
    }
    x[j].keep_packed();
  }
  const float total = row_sum<V>(part, sums[slot], warp_in_row);
  const float rms = __fsqrt_rn(__fadd_rn(__fdiv_rn(total, static_cast<float>(dim)), epsilon));
  const float rstd = __fdiv_rn(1.0f, rms);
  if (!live)
  {
    return;
  }
  if (c0 == 0 && rms_cache != nullptr)
  {
    rms_cache[r] = rms;
  }
  T *dst = output + static_cast<int64_t>(r) * dim;
#pragma unroll
  for (int j = 0; j < STRIPES; ++j)
  {
    const int c = c0 + 256 * j;
    if (c < dim)
    {
      const Gammas<V> g = load_gamma<V>(gamma, c);
      float v[V];
#pragma unroll
      for (int i = 0; i < V; ++i)
      {
        v[i] = __fmul_rn(__fmul_rn(x[j].get(i), rstd), g.e[i]);
      }
      Piece<T, V> y;
      y.set(v);
      *reinterpret_cast<Piece<T, V> *>(dst + c) = y;
    }
  }
}

template <typename T, int V, int STRIPES>
void rows_fwd_inst(const void *input, const float *gamma, void *output, float *rms_cache, float epsilon, int rows,
                   int dim, cudaStream_t s)
{
  launch_dependent(rmsnorm_fwd_rows_kernel<T, V, STRIPES>, dim3(static_cast<unsigned>((rows + V - 1) / V)),
                   dim3(kNormThreads), 0, s, static_cast<const T *>(input), gamma, static_cast<T *>(output), rms_cache,
                   epsilon, rows, dim);
}

template <typename T>
void rows_fwd(const void *input, const float *gamma, void *output, float *rms_cache, float epsilon, int rows, int dim,
              cudaStream_t s)
{
  constexpr int WIDE = 16 / static_cast<int>(sizeof(T));
  // 16-byte pieces need eight (fp32: four) rows a CTA and up to 96 registers of row: from a CTA per SM on
  if (rows >= 148 * WIDE && dim <= 256 * 24)
  {
    if (dim <= 256 * 8)
    {
      rows_fwd_inst<T, WIDE, 8>(input, gamma, output, rms_cache, epsilon, rows, dim, s);
    }
    else if (dim <= 256 * 16)
    {
      rows_fwd_inst<T, WIDE, 16>(input, gamma, output, rms_cache, epsilon, rows, dim, s);
    }
    else
    {
      rows_fwd_inst<T, WIDE, 24>(input, gamma, output, rms_cache, epsilon, rows, dim, s);
    }
  }
  else if (dim <= 256 * 16)
  {
    rows_fwd_inst<T, 2, 16>(input, gamma, output, rms_cache, epsilon, rows, dim, s);
  }
  else if (dim <= 256 * 32)
  {
    rows_fwd_inst<T, 2, 32>(input, gamma, output, rms_cache, epsilon, rows, dim, s);
  }
  else
  {
    rows_fwd_inst<T, 2, 64>(input, gamma, output, rms_cache, epsilon, rows, dim, s);
  }
}

// dy * gamma - x_hat * sum_term is evaluated as fma(dy, gamma, -(x_hat * sum_term)): the fusion the reference
// build makes of that expression (of the three possible evaluations only this one reproduces its dx bit for bit,
// fp32 and bf16).
template <typename T>
__global__ void __launch_bounds__(kNormThreads)
rmsnorm_bwd_kernel(const T *__restrict__ grad_output, const T *__restrict__ input, const float *__restrict__ gamma,
                   const float *__restrict__ rms_cache, T *__restrict__ grad_input, float *__restrict__ grad_gamma,
                   int rows, int dim, int vec)
{
  extern __shared__ __align__(16) unsigned char norm_smem[];
  __shared__ float warp_sums[kNormWarps + 1];
  T *xrow = reinterpret_cast<T *>(norm_smem);
  T *grow = xrow + dim;
  float gg[kNormMaxPerThread];
#pragma unroll
  for (int j = 0; j < kNormMaxPerThread; ++j)
  {
    gg[j] = 0.0f;
  }
  for (int r = blockIdx.x; r < rows; r += gridDim.x)
  {
    __syncthreads();
    row_in<kNormThreads>(xrow, input + static_cast<int64_t>(r) * dim, dim, vec != 0);
    row_in<kNormThreads>(grow, grad_output + static_cast<int64_t>(r) * dim, dim, vec != 0);
    __syncthreads();
    const float rstd = __fdiv_rn(1.0f, __ldg(rms_cache + r));
    float local = 0.0f;
    for (int c = threadIdx.x; c < dim; c += kNormThreads)
    {
      const float x_hat = __fmul_rn(nf<T>(xrow[c]), rstd);
      local = __fmaf_rn(__fmul_rn(nf<T>(grow[c]), __ldg(gamma + c)), x_hat, local);
    }
    const float sum_term = __fdiv_rn(block_sum(local, warp_sums), static_cast<float>(dim));
#pragma unroll
    for (int j = 0; j < kNormMaxPerThread; ++j)
    {
      const int c = threadIdx.x + j * kNormThreads;
      if (c < dim)
      {
        const float x_hat = __fmul_rn(nf<T>(xrow[c]), rstd);
        const float dy = nf<T>(grow[c]);
        const float g = __ldg(gamma + c);
        const float inner = __fmaf_rn(dy, g, -__fmul_rn(x_hat, sum_term));
        gg[j] = __fmaf_rn(dy, x_hat, gg[j]);
        xrow[c] = nt<T>(__fmul_rn(rstd, inner));
      }
    }
    __syncthreads();
    row_out<kNormThreads>(grad_input + static_cast<int64_t>(r) * dim, xrow, dim, vec != 0);
  }
  if (grad_gamma != nullptr)
  {
#pragma unroll
    for (int j = 0; j < kNormMaxPerThread; ++j)
    {
      const int c = threadIdx.x + j * kNormThreads;
      if (c < dim)
      {
        atomicAdd(grad_gamma + c, gg[j]);
      }
    }
  }
}

// Backward with rows in registers (V = 2: four warps a row, two rows at a time per CTA, two CTAs per SM).  The next
// row's pieces are loaded while the current one is worked on where the registers allow it.  grad_gamma: 32 sums a
// thread at 4096 columns, the CTA's two halves meet in shared memory and leave as one two-wide reduction per thread
// and column pair; with one atomic per column and 888 CTAs those were a third of the time (4096 x 4096 bf16: 60 us,
// now 31).
template <typename T, int STRIPES>
__global__ void __launch_bounds__(kNormThreads, 2)
rmsnorm_bwd_rows_kernel(const T *grad_output, const T *input, const float *gamma, const float *rms_cache,
                        T *grad_input, float *grad_gamma, int rows, int dim, int gamma_vec)
{
  // (launched ahead of the previous kernel's end; the next kernel may follow once that one is complete.  gamma's address
  // comes out of the wait, so that its invariant loads stay behind it)
  asm volatile("griddepcontrol.wait;" : "+l"(gamma)::"memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  constexpr int V = 2;
  constexpr bool PREFETCH = STRIPES * sizeof(T) <= 32;
  __shared__ float sums[V][8];
  extern __shared__ __align__(16) unsigned char norm_smem[];   // [dim] sums of the second half
  const int slot = threadIdx.x >> 7;
  const int warp_in_row = (threadIdx.x >> 5) & 3;
  const int c0 = (threadIdx.x & 127) * V;
  Piece<T, V> x[STRIPES], d[STRIPES];
  float gg[STRIPES][V];
#pragma unroll
  for (int j = 0; j < STRIPES; ++j)
  {
    gg[j][0] = gg[j][1] = 0.0f;
  }
  auto load = [&](int r, Piece<T, V> (&xr)[STRIPES], Piece<T, V> (&dr)[STRIPES])
  {
    const bool live = r < rows;
    const int64_t base = static_cast<int64_t>(live ? r : 0) * dim;
#pragma unroll
    for (int j = 0; j < STRIPES; ++j)
    {
      const int c = c0 + 256 * j;
      xr[j] = (live && c < dim) ? *reinterpret_cast<const Piece<T, V> *>(input + base + c) : zero_piece<T, V>();
      dr[j] = (live && c < dim) ? *reinterpret_cast<const Piece<T, V> *>(grad_output + base + c) : zero_piece<T, V>();
    }
  };
  const int step = gridDim.x * V;
  if (PREFETCH)
  {
    load(blockIdx.x * V + slot, x, d);
  }
  // every thread makes the same trips: the row sum has barriers
  for (int r0 = blockIdx.x * V; r0 < rows; r0 += step)
  {
    const int r = r0 + slot;
    const bool live = r < rows;
    Piece<T, V> nx[STRIPES], nd[STRIPES];
    if (PREFETCH)
    {
      load(r + step, nx, nd);
    }
    else
    {
      load(r, x, d);
    }
    const float rstd = __fdiv_rn(1.0f, live ? rms_cache[r] : 1.0f);
    float part[V] = {0.0f, 0.0f};
#pragma unroll
    for (int j = 0; j < STRIPES; ++j)
    {
      const int c = c0 + 256 * j;
      if (c < dim)
      {
        const Gammas<V> g = load_gamma<V>(gamma, c);
#pragma unroll
        for (int i = 0; i < V; ++i)
        {
          part[i] = __fmaf_rn(__fmul_rn(d[j].get(i), g.e[i]), __fmul_rn(x[j].get(i), rstd), part[i]);
        }
      }
      x[j].keep_packed();
      d[j].keep_packed();
    }
    const float sum_term = __fdiv_rn(row_sum<V>(part, sums[slot], warp_in_row), static_cast<float>(dim));
    T *dst = grad_input + static_cast<int64_t>(live ? r : 0) * dim;
#pragma unroll
    for (int j = 0; j < STRIPES; ++j)
    {
      const int c = c0 + 256 * j;
      if (live && c < dim)
      {
        const Gammas<V> g = load_gamma<V>(gamma, c);
        float v[V];
#pragma unroll
        for (int i = 0; i < V; ++i)
        {
          const float dv = d[j].get(i);
          const float h = __fmul_rn(x[j].get(i), rstd);
          gg[j][i] = __fmaf_rn(dv, h, gg[j][i]);
          v[i] = __fmul_rn(rstd, __fmaf_rn(dv, g.e[i], -__fmul_rn(h, sum_term)));
        }
        Piece<T, V> o;
        o.set(v);
        *reinterpret_cast<Piece<T, V> *>(dst + c) = o;
      }
    }
    if (PREFETCH)
    {
#pragma unroll
      for (int j = 0; j < STRIPES; ++j)
      {
        x[j] = nx[j];
        d[j] = nd[j];
      }
    }
  }
  if (grad_gamma == nullptr)
  {
    return;
  }
  float2 *half = reinterpret_cast<float2 *>(norm_smem);
  if (slot == 1)
  {
#pragma unroll
    for (int j = 0; j < STRIPES; ++j)
    {
      const int c = c0 + 256 * j;
      if (c < dim)
      {
        half[c >> 1] = make_float2(gg[j][0], gg[j][1]);
      }
    }
  }
  __syncthreads();
  if (slot == 0)
  {
#pragma unroll
    for (int j = 0; j < STRIPES; ++j)
    {
      const int c = c0 + 256 * j;
      if (c < dim)
      {
        const float2 o = half[c >> 1];
        const float a = gg[j][0] + o.x;
        const float b = gg[j][1] + o.y;
        if (gamma_vec)
        {
          asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(grad_gamma + c), "f"(a), "f"(b) : "memory");
        }
        else
        {
          atomicAdd(grad_gamma + c, a);
          atomicAdd(grad_gamma + c + 1, b);
        }
      }
    }
  }
}

template <typename T, int STRIPES>
void rows_bwd_inst(const void *dy, const void *x, const float *gamma, const float *rms, void *dx, float *grad_gamma,
                   int rows, int dim, cudaStream_t s)
{
  const int pairs = (rows + 1) / 2;
  const int grid = pairs < 148 * 2 ? pairs : 148 * 2;
  launch_dependent(rmsnorm_bwd_rows_kernel<T, STRIPES>, dim3(static_cast<unsigned>(grid)), dim3(kNormThreads),
                   static_cast<size_t>(dim) * 4, s, static_cast<const T *>(dy), static_cast<const T *>(x), gamma, rms,
                   static_cast<T *>(dx), grad_gamma, rows, dim, (reinterpret_cast<uintptr_t>(grad_gamma) & 7u) == 0 ? 1 : 0);
}

template <typename T>
void rows_bwd(const void *dy, const void *x, const float *gamma, const float *rms, void *dx, float *grad_gamma,
              int rows, int dim, cudaStream_t s)
{
  if (dim <= 256 * 8)
  {
    rows_bwd_inst<T, 8>(dy, x, gamma, rms, dx, grad_gamma, rows, dim, s);
  }
  else if (dim <= 256 * 16)
  {
    rows_bwd_inst<T, 16>(dy, x, gamma, rms, dx, grad_gamma, rows, dim, s);
  }
  else if constexpr (sizeof(T) == 2)
  {
    rows_bwd_inst<T, 24>(dy, x, gamma, rms, dx, grad_gamma, rows, dim, s);
  }
}

// Dynamic shared memory that needs no attribute: the static part counts toward the 48 KB, too (fp32 rows of 6144 backward are
// 48 KB by themselves)
constexpr size_t kNormPlainSmem = 47 * 1024;

int norm_grid(int rows, int ctas_per_sm)
{
  const int cap = 148 * ctas_per_sm;
  return rows < cap ? rows : cap;
}

bool rows_vectorizable(const void *a, const void *b, int dim, size_t elem)
{
  return (dim * elem) % 16 == 0 && (reinterpret_cast<uintptr_t>(a) & 15u) == 0 &&
         (reinterpret_cast<uintptr_t>(b) & 15u) == 0;
}

}  // namespace

int launch_rmsnorm_fwd(const void *input, const float *gamma, void *output, float *rms_cache, float epsilon, int dtype,
                       int rows, int dim, cudaStream_t s)
{
  if (rows <= 0)
  {
    return CAIFQ_OK;
  }
  const size_t elem = (dtype == CAIFQ_F32) ? 4 : 2;
  const int vec = rows_vectorizable(input, output, dim, elem) ? 1 : 0;
  if (vec != 0 && dim <= 256 * 64 && (reinterpret_cast<uintptr_t>(gamma) & 15u) == 0)
  {
    if (dtype == CAIFQ_F32)
    {
      rows_fwd<float>(input, gamma, output, rms_cache, epsilon, rows, dim, s);
    }
    else if (dtype == CAIFQ_F16)
    {
      rows_fwd<__half>(input, gamma, output, rms_cache, epsilon, rows, dim, s);
    }
    else
    {
      rows_fwd<__nv_bfloat16>(input, gamma, output, rms_cache, epsilon, rows, dim, s);
    }
    CAIFQ_CHECK_LAUNCH();
    return CAIFQ_OK;
  }
  const size_t smem = static_cast<size_t>(dim) * elem;
  if (smem > 96 * 1024)
  {
    set_error("rmsnorm: rows of %d elements do not fit the row buffer", dim);
    return CAIFQ_ERR_UNSUPPORTED;
  }
#define CAIFQ_NORM_FWD(T)                                                                                        \
  {                                                                                                               \
    if (smem > kNormPlainSmem)                                                                                         \
    {                                                                                                             \
      cudaFuncSetAttribute(rmsnorm_fwd_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024);        \
    }                                                                                                             \
    rmsnorm_fwd_kernel<T><<<norm_grid(rows, 8), kNormThreads, smem, s>>>(static_cast<const T *>(input), gamma,    \
                                                                         static_cast<T *>(output), rms_cache,     \
                                                                         epsilon, rows, dim, vec);                \
  }
  if (dtype == CAIFQ_F32)
    CAIFQ_NORM_FWD(float)
  else if (dtype == CAIFQ_F16)
    CAIFQ_NORM_FWD(__half)
  else
    CAIFQ_NORM_FWD(__nv_bfloat16)
#undef CAIFQ_NORM_FWD
  CAIFQ_CHECK_LAUNCH();
  return CAIFQ_OK;
}

int launch_rmsnorm_bwd(const void *grad_output, const void *input, const float *gamma, const float *rms_cache,
                       void *grad_input, float *grad_gamma, int dtype, int rows, int dim, cudaStream_t s)
{
  if (rows <= 0)
  {
    return CAIFQ_OK;
  }
  const size_t elem = (dtype == CAIFQ_F32) ? 4 : 2;
  const size_t smem = 2 * static_cast<size_t>(dim) * elem;
  if (smem > 96 * 1024 || dim > kNormThreads * kNormMaxPerThread)
  {
    set_error("rmsnorm backward: rows of %d elements are too long", dim);
    return CAIFQ_ERR_UNSUPPORTED;
  }
  const int vec = (rows_vectorizable(input, grad_input, dim, elem) && rows_vectorizable(grad_output, grad_output, dim, elem))
                      ? 1
                      : 0;
  // (fp32 rows of more than 4096 columns do not fit the registers beside their share of grad_gamma)
  if (vec != 0 && dim <= 256 * (elem == 4 ? 16 : 24) && (reinterpret_cast<uintptr_t>(gamma) & 15u) == 0)
  {
    if (dtype == CAIFQ_F32)
    {
      rows_bwd<float>(grad_output, input, gamma, rms_cache, grad_input, grad_gamma, rows, dim, s);
    }
    else if (dtype == CAIFQ_F16)
    {
      rows_bwd<__half>(grad_output, input, gamma, rms_cache, grad_input, grad_gamma, rows, dim, s);
    }
    else
    {
      rows_bwd<__nv_bfloat16>(grad_output, input, gamma, rms_cache, grad_input, grad_gamma, rows, dim, s);
    }
    CAIFQ_CHECK_LAUNCH();
    return CAIFQ_OK;
  }
#define CAIFQ_NORM_BWD(T)                                                                                        \
  {                                                                                                               \
    if (smem > kNormPlainSmem)                                                                                         \
    {                                                                                                             \
      cudaFuncSetAttribute(rmsnorm_bwd_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024);        \
    }                                                                                                             \
    rmsnorm_bwd_kernel<T><<<norm_grid(rows, 4), kNormThreads, smem, s>>>(                                         \
        static_cast<const T *>(grad_output), static_cast<const T *>(input), gamma, rms_cache,                     \
        static_cast<T *>(grad_input), grad_gamma, rows, dim, vec);                                                \
  }
  if (dtype == CAIFQ_F32)
    CAIFQ_NORM_BWD(float)
  else if (dtype == CAIFQ_F16)
    CAIFQ_NORM_BWD(__half)
  else
    CAIFQ_NORM_BWD(__nv_bfloat16)
#undef CAIFQ_NORM_BWD
  CAIFQ_CHECK_LAUNCH();
  return CAIFQ_OK;
}

}  // namespace caifq
