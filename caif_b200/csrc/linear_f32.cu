// Frozen-linear products of fp32 activations with int8 / int4 weights, fp32 compute (the layers' default element type):
//
//   forward : C[m, out] = A[m, in]  . W_deq[out, in]^T     (ForwardImpl,  src/caif_device_frozen_linear.cpp:381-524)
//   backward: C[m, in]  = A[m, out] . W_deq[out, in]       (BackwardImpl, src/caif_device_frozen_linear.cpp:526-660)
//
// The fp32-FMA kernel is bound by 37 TFLOP/s of FMA at best.  Here an fp32 activation goes to the bf16 tensor core as three
// terms, hi + mid + lo, eight bits of its mantissa each: exact.  Codes are exact in bf16, so every product is exact and the
// sums run in fp32: the terms of 64 elements of k in one accumulation chain, the chains added with IEEE additions, as good
// as the FMA chain they replace.  The scale never enters an operand that would round it: int8's multiplies the final sum;
// int4's multiplies the fp32 sum of a chain in the forward product (a chain lies in one group) and the fp32 gradient before
// its split in dX (a column tile lies in one group).
// (Four signed bytes of a fixed-point activation were measured too: mma.sync runs integers at a quarter of the bf16 rate
// here, and elements far below their block's largest lose bits.)
//
// A CTA owns a tile of 64 x 64 and takes 64 of k at a time (four warps); the next ones are on their way from global memory
// while the current ones are multiplied.  Up to 16 rows the tile is 16 x 64 and 128 of k (eight warps): such a call is a chain
// of latencies, and the next block is also split while the current one is multiplied (that cost the larger tile more than
// it gave: 4096 -> 4096, 64 rows, 42 us against 35).  Calls with few tiles split k over the CTAs of a cluster, whose partial
// tiles meet through distributed shared memory in rank order: no scratch, no atomics, the same bits every time.
// The first codes are read before the previous kernel's end.  The next kernel is let in when the main loop is over: its
// clusters would otherwise share SMs with this one's while others have none.
// us a call, int8, forward / dX, tiles of 64 rows and plain launches / now: 1024 -> 1024, 1 row 6.4, 6.9 / 4.2, 4.2; 4096 ->
// 4096, 3 rows 28.7, 35.7 / 16.4, 16.1; 3712 -> 768, 16 rows 11.7, 8.7 / 6.9, 6.1.
#include <atomic>

#include "common.cuh"

namespace caifq
{

namespace
{

// more than 16 rows: 64 x 64, 64 of k, four warps of 32 x 32
constexpr int FM = 64;
constexpr int FN = 64;
constexpr int FK = 64;
constexpr int F_THREADS = 128;
constexpr uint32_t F_PLANE = FM * FK * 2;   // bytes of one bf16 operand plane
constexpr int F_PLANES = 3;
// up to 16 rows: 16 x 64, 128 of k in two accumulation chains, eight warps of 16 x 8
constexpr int RM = 16;
constexpr int R_FK = 128;
constexpr int CHAIN = 64;
constexpr int R_THREADS = 256;
constexpr uint32_t R_A_PLANE = RM * R_FK * 2;
constexpr uint32_t R_BUFFER = F_PLANES * R_A_PLANE + FN * R_FK * 2;

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

// The activations, whose address comes out of the wait for the previous kernel: such a load cannot move ahead of the wait, but
// it can move past the stores to shared memory (a plain one cannot, 1024 rows of int4 dX, 4096 -> 4096: 535 us against 510)
__device__ __forceinline__ float4 f32_ldg(const float *p)
{
  float4 v;
  asm("ld.global.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  return v;
}

__device__ __forceinline__ void f32_sts2(uint32_t addr, uint32_t a, uint32_t b)
{
  asm volatile("st.shared.v2.u32 [%0], {%1,%2};" ::"r"(addr), "r"(a), "r"(b) : "memory");
}

__device__ __forceinline__ void f32_sts4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d)
{
  asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

// sixteen-byte chunks of a row of `pitch` bytes XOR the row
__device__ __forceinline__ uint32_t f32_at(uint32_t base, int row, int chunk, int pitch)
{
  return base + static_cast<uint32_t>(row * pitch + ((chunk ^ (row & 7)) << 4));
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

// The partial tiles of a cluster's CTAs, [TILE][FN] each, become the result.
template <int TILE, int THREADS, bool I4>
__device__ __forceinline__ void f32_finish(const F32Params &p, float *part, int64_t m0, int n0, int rank)
{
  const int tid = threadIdx.x;
  if (p.splits > 1)
  {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
  else
  {
    __syncthreads();
  }
  const int rows_each = TILE / p.splits;
  const float tensor_scale = (!I4 && p.scales != nullptr) ? __ldg(static_cast<const float *>(p.scales)) : 1.0f;
  for (int idx = tid; idx < rows_each * (FN / 4); idx += THREADS)
  {
    const int r = rank * rows_each + idx / (FN / 4);
    const int c = (idx % (FN / 4)) * 4;
    if (m0 + r >= p.m)
    {
      continue;
    }
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
  if (p.splits > 1)
  {
    // nobody leaves while another CTA may still read its partial tile
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
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
  const float *src = p.a;
  auto load = [&](int kb, bool with_a, bool with_w)
  {
    const int k0 = kb * FK;
#pragma unroll
    for (int i = 0; i < A_LOADS; ++i)
    {
      const int idx = tid + i * F_THREADS;
      const int64_t row = m0 + (idx >> 4);
      const int k = k0 + (idx & 15) * 4;
      if (with_a)
      {
        ra[i] = row < p.m ? f32_ldg(src + row * p.k_total + k) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
      if constexpr (I4 && BWD)
      {
        if (with_w)
        {
#pragma unroll
          for (int e = 0; e < 4; ++e)
          {
            rk[i][e] = __half2float(__ldg(scales4 + static_cast<int64_t>(k + e) * groups_per_row + n0 / p.group_size));
          }
        }
      }
    }
    if (!with_w)
    {
      return;
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
      const uint32_t at = f32_at(a_base, row, c4 >> 1, 128) + static_cast<uint32_t>((c4 & 1) * 8);
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
        asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(f32_at(b_base, row, piece * OUT + o, 128)), "r"(v.x),
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
  // The weight does not depend on earlier work in the stream: its first tile is on the way before the wait for it (not where
  // its scales multiply the activations: apart, those loads cost 4 % at 512 rows and more)
  constexpr bool EARLY = !(I4 && BWD);
  if (EARLY && kb_begin < kb_end)
  {
    load(kb_begin, false, true);
  }
  asm volatile("griddepcontrol.wait;" : "+l"(src)::"memory");
  if (kb_begin < kb_end)
  {
    load(kb_begin, true, !EARLY);
  }
  for (int kb = kb_begin; kb < kb_end; ++kb)
  {
    stage();
    __syncthreads();
    if (kb + 1 < kb_end)
    {
      load(kb + 1, true, true);
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
            f32_ldmatrix_trans(r, f32_at(b_base, k16 * 16 + (mat & 1) * 8 + (lane & 7), (wn >> 3) + 2 * h + (mat >> 1), 128));
          }
          else
          {
            f32_ldmatrix(r, f32_at(b_base, wn + 16 * h + (mat >> 1) * 8 + (lane & 7), k16 * 2 + (mat & 1), 128));
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
            f32_ldmatrix(a, f32_at(a_base + plane * F_PLANE, wm + 16 * i + (lane & 15), k16 * 2 + (lane >> 4), 128));
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

  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
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
  f32_finish<FM, F_THREADS, I4>(p, part, m0, n0, rank);
}

template <bool I4, bool BWD>
__global__ void __launch_bounds__(R_THREADS, 2) linear_f32_rows_kernel(const F32Params p)
{
  constexpr int FK = R_FK;
  constexpr int THREADS = R_THREADS;
  constexpr uint32_t A_PLANE = R_A_PLANE;
  constexpr int A_LOADS = RM * FK / 4 / THREADS;   // 16-byte pieces of A per thread, side by side across the threads
  constexpr int A_PITCH = FK * 2;
  constexpr int B_PITCH = BWD ? FN * 2 : FK * 2;   // the code tile lies as in memory: [n][k] forward, [k][n] dX
  extern __shared__ __align__(128) uint8_t f32_tiles[];   // two buffers: three planes of A, the codes
  __shared__ float s_col[2][FK / CHAIN][FN];   // int4 forward: the chains' group scales of every column
  __shared__ float s_k[2][FK];       // int4 dX: the scales of the block's k
  const int tid = threadIdx.x;
  const int warp = tid >> 5;
  const int lane = tid & 31;
  const int64_t m0 = static_cast<int64_t>(blockIdx.y) * RM;
  const int n0 = static_cast<int>(blockIdx.x) * FN;
  const int rank = static_cast<int>(blockIdx.z);
  const int num_kb = (p.k_total + FK - 1) / FK;
  const int kb_begin = (num_kb * rank) / p.splits;
  const int kb_end = (num_kb * (rank + 1)) / p.splits;
  const int groups_per_row = I4 ? p.in_dim / p.group_size : 1;
  const __half *scales4 = static_cast<const __half *>(p.scales);
  const uint32_t base = f32_smem(f32_tiles);

  // ---- a block of k on its way, in registers
  float4 ra[A_LOADS];
  constexpr int B_ROWS = BWD ? FK : FN;
  constexpr int B_PIECES = (BWD ? FN : FK) / (I4 ? 32 : 16);              // sixteen-byte pieces of a row of codes
  constexpr int B_LOADS = B_ROWS * B_PIECES / THREADS;
  static_assert(B_ROWS * B_PIECES % THREADS == 0, "whole pieces for every thread");
  uint4 rb[B_LOADS];
  float rs = 1.0f;                // int4 forward: the scale of column tid % FN, chain tid / FN
  const float *src = p.a;
  auto load_a = [&](int kb)
  {
#pragma unroll
    for (int i = 0; i < A_LOADS; ++i)
    {
      const int idx = tid + i * THREADS;
      const int64_t row = m0 + idx / (FK / 4);
      const int k = kb * FK + (idx % (FK / 4)) * 4;
      ra[i] = row < p.m && k < p.k_total ? f32_ldg(src + row * p.k_total + k) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
  };
  auto load_w = [&](int kb)
  {
    const int k0 = kb * FK;
#pragma unroll
    for (int i = 0; i < B_LOADS; ++i)
    {
      const int idx = tid + i * THREADS;
      const int row = idx / B_PIECES;
      const int column = (idx % B_PIECES) * (I4 ? 32 : 16);
      const int out = BWD ? k0 + row : n0 + row;
      const int in = BWD ? n0 + column : k0 + column;
      const int64_t flat = static_cast<int64_t>(out) * p.in_dim + in;
      rb[i] = (BWD ? out : in) < p.k_total ? __ldg(reinterpret_cast<const uint4 *>(p.codes + (I4 ? flat >> 1 : flat)))
                                           : make_uint4(0u, 0u, 0u, 0u);
    }
    if (I4 && !BWD && tid < FN * (FK / CHAIN))
    {
      const int k = k0 + CHAIN * (tid / FN);
      rs = k < p.k_total
               ? __half2float(__ldg(scales4 + static_cast<int64_t>(n0 + tid % FN) * groups_per_row + k / p.group_size))
               : 0.0f;
    }
  };
  // int4 dX: the scale of element tid of a block of k
  auto load_k_scale = [&](int kb)
  {
    const int k = kb * FK + tid;
    return tid < FK && kb < kb_end && k < p.k_total
               ? __half2float(__ldg(scales4 + static_cast<int64_t>(k) * groups_per_row + n0 / p.group_size))
               : 0.0f;
  };
  auto stage = [&](int buffer)
  {
    const uint32_t a_base = base + static_cast<uint32_t>(buffer) * R_BUFFER;
    const uint32_t b_base = a_base + F_PLANES * A_PLANE;
#pragma unroll
    for (int i = 0; i < A_LOADS; ++i)
    {
      const int idx = tid + i * THREADS;
      const int c4 = idx % (FK / 4);
      float4 v = ra[i];
      if constexpr (I4 && BWD)
      {
        const float *s = s_k[buffer] + 4 * c4;
        v.x *= s[0];
        v.y *= s[1];
        v.z *= s[2];
        v.w *= s[3];
      }
      uint32_t hi[2], mid[2], lo[2];
      f32_split(v.x, v.y, hi[0], mid[0], lo[0]);
      f32_split(v.z, v.w, hi[1], mid[1], lo[1]);
      const uint32_t at = f32_at(a_base, idx / (FK / 4), c4 >> 1, A_PITCH) + static_cast<uint32_t>((c4 & 1) * 8);
      f32_sts2(at, hi[0], hi[1]);
      f32_sts2(at + A_PLANE, mid[0], mid[1]);
      f32_sts2(at + 2 * A_PLANE, lo[0], lo[1]);
    }
#pragma unroll
    for (int i = 0; i < B_LOADS; ++i)
    {
      const int idx = tid + i * THREADS;
      const uint32_t w[4] = {rb[i].x, rb[i].y, rb[i].z, rb[i].w};
      constexpr int OUT = I4 ? 4 : 2;   // sixteen-byte chunks of bf16 per piece
#pragma unroll
      for (int o = 0; o < OUT; ++o)
      {
        const uint4 v = I4 ? f32_int4x8(w[o]) : expand_int8x8(make_uint2(w[(2 * o) & 3], w[(2 * o + 1) & 3]));
        f32_sts4(f32_at(b_base, idx / B_PIECES, (idx % B_PIECES) * OUT + o, B_PITCH), v.x, v.y, v.z, v.w);
      }
    }
    if (I4 && !BWD && tid < FN * (FK / CHAIN))
    {
      s_col[buffer][tid / FN][tid % FN] = rs;
    }
  };

  const int wn = warp * 8;
  float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
  // The weight does not depend on earlier work in the stream: its first tile is on the way before the wait for it
  if (kb_begin < kb_end)
  {
    load_w(kb_begin);
  }
  if constexpr (I4 && BWD)
  {
    const float first = load_k_scale(kb_begin), second = load_k_scale(kb_begin + 1);
    if (tid < FK)
    {
      s_k[0][tid] = first;
      s_k[1][tid] = second;
    }
    __syncthreads();
  }
  asm volatile("griddepcontrol.wait;" : "+l"(src)::"memory");
  if (kb_begin < kb_end)
  {
    load_a(kb_begin);
  }
  auto load_next = [&](int kb)
  {
    if (kb < kb_end)
    {
      load_w(kb);
      load_a(kb);
    }
  };
  if (kb_begin < kb_end)
  {
    stage(0);
    load_next(kb_begin + 1);
    __syncthreads();
  }
  for (int kb = kb_begin; kb < kb_end; ++kb)
  {
    const int parity = (kb - kb_begin) & 1;
    const uint32_t a_base = base + static_cast<uint32_t>(parity) * R_BUFFER;
    const uint32_t b_base = a_base + F_PLANES * A_PLANE;
    float next_scale = 0.0f;
    if constexpr (I4 && BWD)
    {
      next_scale = load_k_scale(kb + 2);
    }
#pragma unroll
    for (int part = 0; part < FK / CHAIN; ++part)
    {
      float chain[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
      for (int k16 = part * (CHAIN / 16); k16 < (part + 1) * (CHAIN / 16); k16 += 2)
      {
        // the codes of 32 of k: two MMAs' operands
        uint32_t b[4];
        const int mat = lane >> 3;
        if constexpr (BWD)
        {
          f32_ldmatrix_trans(b, f32_at(b_base, k16 * 16 + mat * 8 + (lane & 7), wn >> 3, B_PITCH));
        }
        else
        {
          f32_ldmatrix(b, f32_at(b_base, wn + (lane & 7), k16 * 2 + mat, B_PITCH));
        }
#pragma unroll
        for (int h = 0; h < 2; ++h)
        {
#pragma unroll
          for (int plane = F_PLANES - 1; plane >= 0; --plane)   // small terms first
          {
            uint32_t a[4];
            f32_ldmatrix(a, f32_at(a_base + static_cast<uint32_t>(plane) * A_PLANE, lane & 15, (k16 + h) * 2 + (lane >> 4), A_PITCH));
            f32_mma(chain, a, b[2 * h], b[2 * h + 1]);
          }
        }
      }
      const float *col = &s_col[parity][part][wn + 2 * (lane & 3)];
#pragma unroll
      for (int e = 0; e < 4; ++e)
      {
        acc[e] = (I4 && !BWD) ? fmaf(col[e & 1], chain[e], acc[e]) : acc[e] + chain[e];
      }
    }
    if constexpr (I4 && BWD)
    {
      if (tid < FK)
      {
        s_k[parity][tid] = next_scale;   // (read last for this block's split, before the last barrier)
      }
    }
    if (kb + 1 < kb_end)
    {
      stage(parity ^ 1);
      load_next(kb + 2);
    }
    __syncthreads();
  }

  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  float *part = reinterpret_cast<float *>(f32_tiles);   // (everything in the buffers has been used)
  const int r = lane >> 2;
  const int c = wn + 2 * (lane & 3);
  *reinterpret_cast<float2 *>(part + r * FN + c) = make_float2(acc[0], acc[1]);
  *reinterpret_cast<float2 *>(part + (r + 8) * FN + c) = make_float2(acc[2], acc[3]);
  f32_finish<RM, R_THREADS, I4>(p, part, m0, n0, rank);
}

template <bool I4, bool BWD>
int launch_f32_inst(F32Params p, cudaStream_t s)
{
  const bool few = p.m <= RM;
  const int tile = few ? RM : FM;
  auto kernel = few ? linear_f32_rows_kernel<I4, BWD> : linear_f32_kernel<I4, BWD>;
  constexpr int smem = 2 * R_BUFFER;
  static std::atomic<bool> configured[kMaxDevices];
  int dev = 0;
  CAIFQ_CHECK_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices)
  {
    set_error("frozen linear (fp32): device ordinal %d out of range", dev);
    return CAIFQ_ERR_UNSUPPORTED;
  }
  if (!configured[dev].load(std::memory_order_acquire))
  {
    CAIFQ_CHECK_CUDA(cudaFuncSetAttribute(linear_f32_rows_kernel<I4, BWD>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    configured[dev].store(true, std::memory_order_release);
  }
  const unsigned nt = static_cast<unsigned>(p.n_total / FN);
  const unsigned mt = static_cast<unsigned>((p.m + tile - 1) / tile);
  // k is split until the SMs hold two CTAs each, as long as a CTA keeps two blocks of 64 to overlap; the smaller tile's CTAs
  // are cheaper to have fewer of (4096 -> 4096, one row: 17.5 us with four a tile, 19.6 with eight)
  const int sms = device_sm_count();
  const int64_t fill = few ? sms : 2 * sms - 1;
  p.splits = 1;
  while (p.splits < 8 && static_cast<int64_t>(nt) * mt * p.splits <= fill && p.k_total / 64 >= 4 * p.splits)
  {
    p.splits *= 2;
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(nt, mt, static_cast<unsigned>(p.splits));
  cfg.blockDim = dim3(few ? R_THREADS : F_THREADS);
  cfg.dynamicSmemBytes = few ? smem : 0;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = static_cast<unsigned>(p.splits);
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  // codes written just ahead in this stream by one of the library's own calls: a plain launch orders the early loads
  // behind that kernel.  64-row tiles of more CTAs than SMs are launched plainly too: while the previous kernel still has
  // its SMs the others get two CTAs each (3712 <- 768, 64 rows, 232 CTAs: 11.1 us, plainly 9.8).
  const bool dependent = dependent_launches() && !take_codes_written(s) && (few || static_cast<int64_t>(nt) * mt * p.splits <= sms);
  cfg.numAttrs = dependent ? 2 : 1;
  CAIFQ_CHECK_CUDA(cudaLaunchKernelEx(&cfg, kernel, p));
  return CAIFQ_OK;
}

}  // namespace

bool f32_supported(const LinearArgs &g)
{
  const caifq_weight &w = g.w;
  const int n_total = g.backward ? w.in_dim : w.out_dim;
  const int k_total = g.backward ? w.out_dim : w.in_dim;
  if (g.a_dtype != CAIFQ_F32 || g.compute_dtype != CAIFQ_F32 || g.a_prescale != 1.0f || g.m < 1 || g.num_peers != 0 ||
      g.num_more != 0 || (n_total % 64) != 0 || (k_total % 64) != 0 || g.m > static_cast<int64_t>(65535) * 64 ||
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
  if (g.w.storage == CAIFQ_I4)
  {
    return g.backward ? launch_f32_inst<true, true>(p, s) : launch_f32_inst<true, false>(p, s);
  }
  return g.backward ? launch_f32_inst<false, true>(p, s) : launch_f32_inst<false, false>(p, s);
}

}  // namespace caifq
