// Frozen-linear products of fp32 activations with int8 / int4 weights, fp32 compute (the layers' default element type):
//
//   forward : C[m, out] = A[m, in]  . W_deq[out, in]^T     (ForwardImpl,  src/caif_device_frozen_linear.cpp:381-524)
//   backward: C[m, in]  = A[m, out] . W_deq[out, in]       (BackwardImpl, src/caif_device_frozen_linear.cpp:526-660)
//
// The fp32-FMA kernel these calls ran on is bound by 37 TFLOP/s of FMA at best and reached 12; small calls were a
// handful of its CTAs walking all of k (1024 x 1024, m = 64: 81 us forward, 107 us dX).  Here an fp32 activation goes
// to the bf16 tensor core as three terms, hi + mid + lo, eight bits of its mantissa each: exact.  Codes are exact in
// bf16, so every product is exact and the sums run in fp32: the terms of 64 elements of k in one accumulation chain,
// the chains added with IEEE additions, as good as the FMA chain they replace.  The scale never enters an operand that
// would round it: int8's multiplies the final sum; int4's multiplies the fp32 sum of a chain in the forward product
// (a chain lies in one group) and the fp32 gradient before its split in dX (a column tile lies in one group).
//
// A CTA of four warps owns a 64 x 64 tile; the next 64 elements of k are on their way from global memory while the
// current ones are multiplied.  Calls with few tiles split k over the CTAs of a cluster, whose partial tiles meet
// through distributed shared memory in rank order: no scratch, no atomics, the same bits every time.
#include "common.cuh"

namespace caifq
{

namespace
{

constexpr int FM = 64;
constexpr int FN = 64;
constexpr int FK = 64;
constexpr int F_THREADS = 128;
constexpr uint32_t F_PLANE = FM * FK * 2;   // bytes of one bf16 operand plane

struct F32Params
{
  const float *a;
  const uint8_t *codes;
  const void *scales;
  void *c;
  int c_dtype;
  int accumulate;
  int64_t m;
  int n_total;
  int k_total;
  int in_dim;
  int group_size;   // int4
  int splits;       // CTAs of a cluster
};

__device__ __forceinline__ uint32_t f32_smem(const void *p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ void f32_mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ void f32_ldmatrix(uint32_t (&r)[4], uint32_t addr)
{
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}

__device__ __forceinline__ void f32_ldmatrix_trans(uint32_t (&r)[4], uint32_t addr)
{
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}

// Two fp32 values -> three bf16x2 terms whose sum they are: the upper halves of the value, of what that leaves, and of
// what that leaves (which has eight bits or fewer).  An infinity is its own first term; a NaN is one in the second at least
// (one whose payload lies in the lower half has the upper half of an infinity).
__device__ __forceinline__ void f32_split(float a, float b, uint32_t &hi, uint32_t &mid, uint32_t &lo)
{
  auto rest = [](float v)
  {
    const float r = v - __uint_as_float(__float_as_uint(v) & 0xFFFF0000u);
    return fabsf(v) == __int_as_float(0x7F800000) ? 0.0f : r;   // (NaN - x: NaN)
  };
  auto upper = [](float x, float y) { return __byte_perm(__float_as_uint(x), __float_as_uint(y), 0x7632); };
  hi = upper(a, b);
  a = rest(a);
  b = rest(b);
  mid = upper(a, b);
  a -= __uint_as_float(__float_as_uint(a) & 0xFFFF0000u);
  b -= __uint_as_float(__float_as_uint(b) & 0xFFFF0000u);
  lo = upper(a, b);
}

// rows of 128 bytes, sixteen-byte chunks XOR the row
__device__ __forceinline__ uint32_t f32_at(uint32_t base, int row, int chunk)
{
  return base + static_cast<uint32_t>(row * 128 + ((chunk ^ (row & 7)) << 4));
}

// eight int4 codes -> bf16 integers in element order
__device__ __forceinline__ uint4 f32_int4x8(uint32_t w)
{
  const uint32_t ev = (w & 0x0F0F0F0Fu) ^ 0x08080808u;
  const uint32_t od = ((w >> 4) & 0x0F0F0F0Fu) ^ 0x08080808u;
  const uint32_t t0 = __byte_perm(ev, od, 0x5140);
  const uint32_t t1 = __byte_perm(ev, od, 0x7362);
  uint32_t o[4] = {__byte_perm(t0, 0x43434343u, 0x4140), __byte_perm(t0, 0x43434343u, 0x4342),
                   __byte_perm(t1, 0x43434343u, 0x4140), __byte_perm(t1, 0x43434343u, 0x4342)};
#pragma unroll
  for (int i = 0; i < 4; ++i)
  {
    asm("sub.rn.bf16x2 %0, %0, %1;" : "+r"(o[i]) : "r"(0x43084308u));   // 136 + q -> q
  }
  return make_uint4(o[0], o[1], o[2], o[3]);
}

template <bool I4, bool BWD>
__global__ void __launch_bounds__(F_THREADS) linear_f32_kernel(const F32Params p)
{
  __shared__ __align__(128) uint8_t sa[3 * F_PLANE];
  __shared__ __align__(128) uint8_t sb[FN * FK * 2];
  __shared__ float s_scale[FN];   // int4 forward: the chain's group scale of every column
  const int tid = threadIdx.x;
  const int warp = tid >> 5;
  const int lane = tid & 31;
  const int64_t m0 = static_cast<int64_t>(blockIdx.y) * FM;
  const int n0 = static_cast<int>(blockIdx.x) * FN;
  const int rank = static_cast<int>(blockIdx.z);
  const int num_kb = p.k_total / FK;
  const int kb_begin = (num_kb * rank) / p.splits;
  const int kb_end = (num_kb * (rank + 1)) / p.splits;
  const int groups_per_row = I4 ? p.in_dim / p.group_size : 1;
  const __half *scales4 = static_cast<const __half *>(p.scales);
  const uint32_t a_base = f32_smem(sa);
  const uint32_t b_base = f32_smem(sb);

  constexpr int A_LOADS = FM * FK / 4 / F_THREADS;                        // 16-byte pieces of A per thread
  constexpr int W_LOADS = (FN * FK / (I4 ? 2 : 1)) / 16 / F_THREADS;      // 16-byte pieces of codes per thread
  float4 ra[A_LOADS];
  uint4 rw[W_LOADS];
  float rs = 1.0f;                // int4: a scale (forward: column tid's; backward: unused)
  float rk[I4 && BWD ? A_LOADS : 1][I4 && BWD ? 4 : 1];   // int4 dX: the scales of the piece's four k
  auto load = [&](int kb)
  {
    const int k0 = kb * FK;
#pragma unroll
    for (int i = 0; i < A_LOADS; ++i)
    {
      const int idx = tid + i * F_THREADS;
      const int64_t row = m0 + (idx >> 4);
      const int k = k0 + (idx & 15) * 4;
      ra[i] = row < p.m ? __ldg(reinterpret_cast<const float4 *>(p.a + row * p.k_total + k)) : make_float4(0.f, 0.f, 0.f, 0.f);
      if constexpr (I4 && BWD)
      {
#pragma unroll
        for (int e = 0; e < 4; ++e)
        {
          rk[i][e] = __half2float(__ldg(scales4 + static_cast<int64_t>(k + e) * groups_per_row + n0 / p.group_size));
        }
      }
    }
    // the code tile: rows are the output features (columns of C forward, k backward), contiguous along `in`
    const int row0 = BWD ? k0 : n0;
    const int col0 = BWD ? n0 : k0;
#pragma unroll
    for (int i = 0; i < W_LOADS; ++i)
    {
      const int idx = tid + i * F_THREADS;
      const int row = I4 ? (idx >> 1) : (idx >> 2);
      const int piece = I4 ? (idx & 1) : (idx & 3);
      const int64_t flat = static_cast<int64_t>(row0 + row) * p.in_dim + col0;
      rw[i] = __ldg(reinterpret_cast<const uint4 *>(p.codes + (I4 ? flat >> 1 : flat) + piece * 16));
    }
    if (I4 && !BWD && tid < FN)
    {
      rs = __half2float(__ldg(scales4 + static_cast<int64_t>(n0 + tid) * groups_per_row + k0 / p.group_size));
    }
  };
  auto stage = [&]()
  {
#pragma unroll
    for (int i = 0; i < A_LOADS; ++i)
    {
      const int idx = tid + i * F_THREADS;
      const int row = idx >> 4;
      const int c4 = idx & 15;
      float4 v = ra[i];
      if constexpr (I4 && BWD)
      {
        v.x *= rk[i][0];
        v.y *= rk[i][1];
        v.z *= rk[i][2];
        v.w *= rk[i][3];
      }
      uint32_t hi[2], mid[2], lo[2];
      f32_split(v.x, v.y, hi[0], mid[0], lo[0]);
      f32_split(v.z, v.w, hi[1], mid[1], lo[1]);
      const uint32_t at = f32_at(a_base, row, c4 >> 1) + static_cast<uint32_t>((c4 & 1) * 8);
      asm volatile("st.shared.v2.u32 [%0], {%1,%2};" ::"r"(at), "r"(hi[0]), "r"(hi[1]) : "memory");
      asm volatile("st.shared.v2.u32 [%0], {%1,%2};" ::"r"(at + F_PLANE), "r"(mid[0]), "r"(mid[1]) : "memory");
      asm volatile("st.shared.v2.u32 [%0], {%1,%2};" ::"r"(at + 2 * F_PLANE), "r"(lo[0]), "r"(lo[1]) : "memory");
    }
#pragma unroll
    for (int i = 0; i < W_LOADS; ++i)
    {
      const int idx = tid + i * F_THREADS;
      const int row = I4 ? (idx >> 1) : (idx >> 2);
      const int piece = I4 ? (idx & 1) : (idx & 3);
      const uint32_t w[4] = {rw[i].x, rw[i].y, rw[i].z, rw[i].w};
      constexpr int OUT = I4 ? 4 : 2;   // sixteen-byte chunks of bf16 per piece
#pragma unroll
      for (int o = 0; o < OUT; ++o)
      {
        const uint4 v = I4 ? f32_int4x8(w[o]) : expand_int8x8(make_uint2(w[(2 * o) & 3], w[(2 * o + 1) & 3]));
        asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(f32_at(b_base, row, piece * OUT + o)), "r"(v.x),
                     "r"(v.y), "r"(v.z), "r"(v.w)
                     : "memory");
      }
    }
    if (I4 && !BWD && tid < FN)
    {
      s_scale[tid] = rs;
    }
  };

  // a warp owns 32 rows x 32 columns
  const int wm = (warp & 1) * 32;
  const int wn = (warp >> 1) * 32;
  const bool rows_live = m0 + wm < p.m;
  float acc[2][4][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
  {
#pragma unroll
    for (int j = 0; j < 4; ++j)
    {
      acc[i][j][0] = acc[i][j][1] = acc[i][j][2] = acc[i][j][3] = 0.0f;
    }
  }
  if (kb_begin < kb_end)
  {
    load(kb_begin);
  }
  for (int kb = kb_begin; kb < kb_end; ++kb)
  {
    stage();
    __syncthreads();
    if (kb + 1 < kb_end)
    {
      load(kb + 1);
    }
    if (rows_live)
    {
      float chain[2][4][4];
#pragma unroll
      for (int i = 0; i < 2; ++i)
      {
#pragma unroll
        for (int j = 0; j < 4; ++j)
        {
          chain[i][j][0] = chain[i][j][1] = chain[i][j][2] = chain[i][j][3] = 0.0f;
        }
      }
#pragma unroll
      for (int k16 = 0; k16 < FK / 16; ++k16)
      {
        uint32_t b[4][2];
        const int mat = lane >> 3;
#pragma unroll
        for (int h = 0; h < 2; ++h)
        {
          uint32_t r[4];
          if (BWD)
          {
            f32_ldmatrix_trans(r, f32_at(b_base, k16 * 16 + (mat & 1) * 8 + (lane & 7), (wn >> 3) + 2 * h + (mat >> 1)));
          }
          else
          {
            f32_ldmatrix(r, f32_at(b_base, wn + 16 * h + (mat >> 1) * 8 + (lane & 7), k16 * 2 + (mat & 1)));
          }
          b[2 * h][0] = r[0];
          b[2 * h][1] = r[1];
          b[2 * h + 1][0] = r[2];
          b[2 * h + 1][1] = r[3];
        }
#pragma unroll
        for (int plane = 2; plane >= 0; --plane)   // small terms first
        {
#pragma unroll
          for (int i = 0; i < 2; ++i)
          {
            uint32_t a[4];
            f32_ldmatrix(a, f32_at(a_base + plane * F_PLANE, wm + 16 * i + (lane & 15), k16 * 2 + (lane >> 4)));
#pragma unroll
            for (int j = 0; j < 4; ++j)
            {
              f32_mma(chain[i][j], a, b[j][0], b[j][1]);
            }
          }
        }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j)
      {
        const float s0 = (I4 && !BWD) ? s_scale[wn + 8 * j + 2 * (lane & 3)] : 1.0f;
        const float s1 = (I4 && !BWD) ? s_scale[wn + 8 * j + 2 * (lane & 3) + 1] : 1.0f;
#pragma unroll
        for (int i = 0; i < 2; ++i)
        {
#pragma unroll
          for (int e = 0; e < 4; ++e)
          {
            acc[i][j][e] = (I4 && !BWD) ? fmaf((e & 1) ? s1 : s0, chain[i][j][e], acc[i][j][e]) : acc[i][j][e] + chain[i][j][e];
          }
        }
      }
    }
    __syncthreads();   // the operand planes are free again
  }

  // partial tile -> shared memory [64][64], where the cluster's CTAs read each other's
  float *part = reinterpret_cast<float *>(sa);
#pragma unroll
  for (int i = 0; i < 2; ++i)
  {
#pragma unroll
    for (int j = 0; j < 4; ++j)
    {
      const int r = wm + 16 * i + (lane >> 2);
      const int c = wn + 8 * j + 2 * (lane & 3);
      *reinterpret_cast<float2 *>(part + r * FN + c) = make_float2(acc[i][j][0], acc[i][j][1]);
      *reinterpret_cast<float2 *>(part + (r + 8) * FN + c) = make_float2(acc[i][j][2], acc[i][j][3]);
    }
  }
  if (p.splits > 1)
  {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
  else
  {
    __syncthreads();
  }
  const int rows_each = FM / p.splits;
  const float tensor_scale = (!I4 && p.scales != nullptr) ? __ldg(static_cast<const float *>(p.scales)) : 1.0f;
  for (int idx = tid; idx < rows_each * (FN / 4); idx += F_THREADS)
  {
    const int r = rank * rows_each + idx / (FN / 4);
    const int c = (idx % (FN / 4)) * 4;
    float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const uint32_t local = f32_smem(part + r * FN + c);
    for (int s = 0; s < p.splits; ++s)
    {
      uint32_t addr = local;
      float4 o;
      if (p.splits > 1)
      {
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(addr) : "r"(local), "r"(s));
      }
      asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(o.x), "=f"(o.y), "=f"(o.z), "=f"(o.w) : "r"(addr));
      v.x += o.x;
      v.y += o.y;
      v.z += o.z;
      v.w += o.w;
    }
    if (m0 + r < p.m)
    {
      const float out[4] = {v.x * tensor_scale, v.y * tensor_scale, v.z * tensor_scale, v.w * tensor_scale};
      const int64_t at = (m0 + r) * p.n_total + n0 + c;
      if (p.c_dtype == CAIFQ_F32 && !p.accumulate)
      {
        *reinterpret_cast<float4 *>(static_cast<float *>(p.c) + at) = make_float4(out[0], out[1], out[2], out[3]);
      }
      else
      {
#pragma unroll
        for (int e = 0; e < 4; ++e)
        {
          float w = out[e];
          if (p.accumulate)
          {
            w = round_through_rt(w, p.c_dtype) + load_as_float(p.c, at + e, p.c_dtype);
          }
          store_from_float(p.c, at + e, p.c_dtype, w);
        }
      }
    }
  }
  if (p.splits > 1)
  {
    // nobody leaves while another CTA may still read its partial tile
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
}

template <bool I4, bool BWD>
int launch_f32_inst(const F32Params &p, dim3 grid, cudaStream_t s)
{
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(F_THREADS);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = static_cast<unsigned>(p.splits);
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  CAIFQ_CHECK_CUDA(cudaLaunchKernelEx(&cfg, linear_f32_kernel<I4, BWD>, p));
  return CAIFQ_OK;
}

}  // namespace

bool f32_supported(const LinearArgs &g)
{
  const caifq_weight &w = g.w;
  const int n_total = g.backward ? w.in_dim : w.out_dim;
  const int k_total = g.backward ? w.out_dim : w.in_dim;
  if (g.a_dtype != CAIFQ_F32 || g.compute_dtype != CAIFQ_F32 || g.a_prescale != 1.0f || g.m < 1 || g.num_peers != 0 ||
      g.num_more != 0 || (n_total % FN) != 0 || (k_total % FK) != 0 || g.m > static_cast<int64_t>(65535) * FM ||
      ((reinterpret_cast<uintptr_t>(g.a) | reinterpret_cast<uintptr_t>(g.c) | reinterpret_cast<uintptr_t>(w.codes)) & 15u) != 0)
  {
    return false;
  }
  if (w.storage == CAIFQ_I8)
  {
    return w.scales == nullptr || w.scheme == CAIFQ_PER_TENSOR;
  }
  return w.storage == CAIFQ_I4 && w.scales != nullptr && w.group_size >= 64 && (w.group_size % 64) == 0 &&
         (w.in_dim % w.group_size) == 0;
}

int launch_linear_f32(const LinearArgs &g, cudaStream_t s)
{
  F32Params p{};
  p.a = static_cast<const float *>(g.a);
  p.codes = static_cast<const uint8_t *>(g.w.codes);
  p.scales = g.w.scales;
  p.c = g.c;
  p.c_dtype = g.c_dtype;
  p.accumulate = g.accumulate ? 1 : 0;
  p.m = g.m;
  p.n_total = g.backward ? g.w.in_dim : g.w.out_dim;
  p.k_total = g.backward ? g.w.out_dim : g.w.in_dim;
  p.in_dim = g.w.in_dim;
  p.group_size = g.w.group_size;
  const unsigned nt = static_cast<unsigned>(p.n_total / FN);
  const unsigned mt = static_cast<unsigned>((g.m + FM - 1) / FM);
  // k is split until the SMs hold two CTAs each, as long as a CTA keeps two blocks of k to overlap
  p.splits = 1;
  while (p.splits < 8 && static_cast<int64_t>(nt) * mt * p.splits < 2 * 148 && p.k_total / FK >= 4 * p.splits)
  {
    p.splits *= 2;
  }
  const dim3 grid(nt, mt, static_cast<unsigned>(p.splits));
  if (g.w.storage == CAIFQ_I4)
  {
    return g.backward ? launch_f32_inst<true, true>(p, grid, s) : launch_f32_inst<true, false>(p, grid, s);
  }
  return g.backward ? launch_f32_inst<false, true>(p, grid, s) : launch_f32_inst<false, false>(p, grid, s);
}

}  // namespace caifq
