// Forward product of a bf16 weight with few rows of bf16 activations, or into few columns:
//
//   y[m, out] = x[m, in] . W[out, in]^T  (+ y)        m <= 16, or any m where out is not a multiple of 128
//
// The float-storage cell of CAIF_DeviceFrozenLinear (src/caif_device_frozen_linear.cpp:381-524) and the router's
// product over the experts (src/caif_device_moe_router.cpp:233-260).  Bound by reading the weight once when it is
// large, by latency when it is small: a router of 64 x 2048 on 16 tokens ran as ONE block of the fp32-FMA kernel that
// walked all of k (191 us; here 7.7 by itself, 4.0 among calls of its kind), by L2 for many rows (16384 tokens: 40 us, the FMA
// kernel 270).  Here a CTA owns NT * 8 output columns and 16 rows, its eight warps split k and stream both operands straight into
// bf16 tensor-core fragments, sixteen bytes a lane and operand (the order of k inside a fragment is the same for both,
// which is all a dot product needs); the eight partial tiles meet in shared memory.  Products are exact in fp32 and
// accumulate in fp32, so fp32 and bf16 compute are the same here.  The tensor core truncates where it adds, so a chain of
// MMAs is 128 k long and the chains meet in IEEE additions: closer to 64 bits than the FMA kernel at every k (one chain a
// warp was not, from k = 8192 on; the many-token kernel's one chain over all of k is five to twelve times further off:
// 12 us for the 16384 tokens, but 2.1e-6 where this and the FMA kernel have 1.3e-7 and 3.9e-7).
#include "common.cuh"

namespace caifq
{

namespace
{

constexpr int kRowsWarps = 8;
constexpr int kRowsChain = 4;   // k-steps of 32 in one chain of MMAs
constexpr unsigned kRowsEarly = 37;   // CTAs (of 256 threads) of a grid that leaves three quarters of the SMs free
constexpr int64_t kRowsMost = 16 * 65535;   // rows of a launch: the grid's second dimension

__device__ __forceinline__ void mma_rows(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1)
{
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// CHAINS: chains whose loads are in flight at a time per warp; CTAS: that an SM must hold, which bounds the registers (0: any)
template <int NT, int CHAINS, int CTAS>
__global__ void __launch_bounds__(kRowsWarps * 32, CTAS)
linear_rows_kernel(const __nv_bfloat16 *x, const __nv_bfloat16 *w, void *y, int y_dtype, int accumulate, int64_t m,
                   int in_dim, int out_dim)
{
  constexpr int UNROLL = kRowsChain * CHAINS;
  __shared__ float part[kRowsWarps][16][NT * 8 + 1];
  // Launched ahead of the previous kernel's end.  A few CTAs let the next kernel in at once (a router's softmax: 0.8 us of an
  // expert layer); of more, it follows as they end: CTAs of the next kernel that are placed earlier share SMs with this one's
  // while others have none (us back to back, let in at once / after the loads / at the end: 14336 -> 1024, 16 rows 19.2 / - /
  // 11.7; -> 1184 11.9 / 13.2 / 11.8; -> 3072 24.5 / 24.1 / 21.2).
  // (The operands' addresses come out of the wait, so that their read-only loads stay behind it.)
  if (gridDim.x * gridDim.y <= kRowsEarly)
  {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  }
  asm volatile("griddepcontrol.wait;" : "+l"(x), "+l"(w)::"memory");
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int g = lane >> 2;
  const int t = lane & 3;
  const int64_t row0 = static_cast<int64_t>(blockIdx.y) * 16;
  const int col0 = static_cast<int>(blockIdx.x) * NT * 8;
  const bool lo_ok = row0 + g < m;
  const bool hi_ok = row0 + g + 8 < m;
  const int steps = in_dim / 32;
  const int begin = (steps * warp) / kRowsWarps;
  const int end = (steps * (warp + 1)) / kRowsWarps;
  const uint4 *x_lo = reinterpret_cast<const uint4 *>(x + (lo_ok ? row0 + g : 0) * in_dim) + t;
  const uint4 *x_hi = reinterpret_cast<const uint4 *>(x + (hi_ok ? row0 + g + 8 : 0) * in_dim) + t;
  const uint4 *w_ptr[NT];
  float sum[NT][4];
#pragma unroll
  for (int nt = 0; nt < NT; ++nt)
  {
    // columns past the last one read it again; they are not stored
    const int col = min(col0 + nt * 8 + g, out_dim - 1);
    w_ptr[nt] = reinterpret_cast<const uint4 *>(w + static_cast<int64_t>(col) * in_dim) + t;
    sum[nt][0] = sum[nt][1] = sum[nt][2] = sum[nt][3] = 0.0f;
  }
  const uint4 zero4 = make_uint4(0u, 0u, 0u, 0u);
  for (int st = begin; st < end; st += UNROLL)
  {
    uint4 xa[UNROLL], xb[UNROLL], wv[UNROLL][NT];
#pragma unroll
    for (int u = 0; u < UNROLL; ++u)
    {
      const bool in = st + u < end;
      xa[u] = (in && lo_ok) ? __ldg(x_lo + (st + u) * 4) : zero4;
      xb[u] = (in && hi_ok) ? __ldg(x_hi + (st + u) * 4) : zero4;
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
      {
        wv[u][nt] = in ? __ldg(w_ptr[nt] + (st + u) * 4) : zero4;
      }
    }
#pragma unroll
    for (int ch = 0; ch < CHAINS; ++ch)
    {
      float c[NT][4] = {};
#pragma unroll
      for (int u = ch * kRowsChain; u < (ch + 1) * kRowsChain; ++u)
      {
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
        {
          mma_rows(c[nt], xa[u].x, xb[u].x, xa[u].y, xb[u].y, wv[u][nt].x, wv[u][nt].y);
          mma_rows(c[nt], xa[u].z, xb[u].z, xa[u].w, xb[u].w, wv[u][nt].z, wv[u][nt].w);
        }
      }
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
      {
#pragma unroll
        for (int i = 0; i < 4; ++i)
        {
          sum[nt][i] += c[nt][i];
        }
      }
    }
  }
#pragma unroll
  for (int nt = 0; nt < NT; ++nt)
  {
    part[warp][g][nt * 8 + 2 * t] = sum[nt][0];
    part[warp][g][nt * 8 + 2 * t + 1] = sum[nt][1];
    part[warp][g + 8][nt * 8 + 2 * t] = sum[nt][2];
    part[warp][g + 8][nt * 8 + 2 * t + 1] = sum[nt][3];
  }
  __syncthreads();
  for (int e = threadIdx.x; e < 16 * NT * 8; e += kRowsWarps * 32)
  {
    const int r = e / (NT * 8);
    const int col = e % (NT * 8);
    if (row0 + r >= m || col0 + col >= out_dim)
    {
      continue;
    }
    float v = 0.0f;
#pragma unroll
    for (int wi = 0; wi < kRowsWarps; ++wi)
    {
      v += part[wi][r][col];
    }
    const int64_t idx = (row0 + r) * out_dim + col0 + col;
    if (accumulate)
    {
      v = round_through_rt(v, y_dtype) + load_as_float(y, idx, y_dtype);
    }
    store_from_float(y, idx, y_dtype, v);
  }
}

}  // namespace

// Few tokens; and any number of them where the output is not made of the tensor-core kernel's 128-column tiles (routers).
bool rows_supported(const LinearArgs &g)
{
  return !g.backward && g.w.storage == CAIFQ_BF16 && g.a_dtype == CAIFQ_BF16 && g.a_prescale == 1.0f && g.m >= 1 &&
         g.m <= ((g.w.out_dim % 128) != 0 ? kRowsMost : 16) && (g.compute_dtype == CAIFQ_F32 || g.compute_dtype == CAIFQ_BF16) &&
         (g.w.in_dim % 32) == 0 &&
         ((reinterpret_cast<uintptr_t>(g.a) | reinterpret_cast<uintptr_t>(g.w.codes)) & 15u) == 0 && g.num_peers == 0 &&
         g.num_more == 0;
}

int launch_linear_rows(const LinearArgs &g, cudaStream_t s)
{
  const unsigned row_tiles = static_cast<unsigned>((g.m + 15) / 16);
  const __nv_bfloat16 *x = static_cast<const __nv_bfloat16 *>(g.a);
  const __nv_bfloat16 *w = static_cast<const __nv_bfloat16 *>(g.w.codes);
  const int acc = g.accumulate ? 1 : 0;
  // 32 columns a CTA share the activations' loads; narrow outputs take 8, for more CTAs, and two chains' loads at a time as
  // long as all CTAs are resident: with 66 registers a thread three are on an SM, and a fourth would be a second wave (us, one
  // row, two chains / one: 4096 -> 3072 4.9 / 6.9, 14336 -> 3552 25 / 31; beyond, 4096 -> 4096 7.7 / 6.9, 14336 -> 4096 49 / 32)
  const int sms = device_sm_count();
  const int wide = (g.w.out_dim + 31) / 32;
  const bool many = wide * row_tiles >= sms;
  const dim3 grid(static_cast<unsigned>(many ? wide : (g.w.out_dim + 7) / 8), row_tiles);
  const unsigned ctas = grid.x * grid.y;
  const bool three = ctas <= 3u * static_cast<unsigned>(sms);
  // 32 columns: 112 registers and two CTAs an SM, except where 80 and three make one wave of what two do not, of rows that share
  // the weight, and where a warp has one trip (us, two / three: 4096 -> 4704, 48 rows 19.1 / 16.9; 14336 -> 3552, 64 rows 89 / 76; 512 ->
  // 1192, 2048 rows 44 / 42; but 4096 -> 9504, 32 rows 30.5 / 35.8; 2048 -> 264, 2048 rows 22 / 26)
  const bool dense = ctas > 2u * static_cast<unsigned>(sms) &&
                     ((three && row_tiles > 2) || g.w.in_dim <= kRowsWarps * kRowsChain * 32);
  auto wide_kernel = dense ? linear_rows_kernel<4, 1, 3> : linear_rows_kernel<4, 1, 0>;
  auto kernel = many ? wide_kernel : (three ? linear_rows_kernel<1, 2, 0> : linear_rows_kernel<1, 1, 0>);
  CAIFQ_CHECK_CUDA(launch_dependent(kernel, grid, dim3(kRowsWarps * 32), 0, s, x, w, g.c, g.c_dtype, acc, g.m, g.w.in_dim,
                                    g.w.out_dim));
  return CAIFQ_OK;
}

}  // namespace caifq
