// Weight-streaming frozen-linear forward for few tokens (decode shapes).
//
//   y[m, out] = x[m, in] . W_deq[out, in]^T  (+ residual)     m <= 16, x bf16, y fp32/bf16/fp16
//
// The call is bound by reading the packed codes once from HBM
// (CAIF_DeviceFrozenLinear::ForwardImpl, src/caif_device_frozen_linear.cpp:381-524,
// does the same product after writing and re-reading an fp32 copy of the whole
// weight, :319-334).  Design:
//   * one CTA per SM owns a contiguous range of rows of the [out, in] code matrix,
//     cut into tiles of 16 rows (the M of the tensor-core instruction).  Copies of
//     the frozen codes and scales never depend on earlier work and start before the
//     kernel waits for the previous one in the stream (programmatic dependent launch);
//   * the warps split the reduction dimension; a warp copies its own pieces of a
//     tile into its own ring (cp.async, 16 bytes a lane) and every lane reads back
//     exactly what it copied, so the main loop has no barrier and no shared
//     address arithmetic;
//   * a lane turns nibbles/bytes of rows g and g+8 into exact bf16 integers with
//     logic ops (no int->float converts), and feeds them as the A operand of bf16
//     tensor-core MMAs against token fragments (B operand) in registers.  Rows too
//     long for the registers are taken in segments of the reduction dimension,
//     one after the other over all tiles of the CTA;
//   * int4 group scales (copied to shared memory ahead of the previous kernel's
//     end) multiply the fp32 partial sum once per 128-element chunk; the int8
//     per-tensor scale multiplies the final sum;
//   * each warp parks its partial sums of every tile (live tokens only) in shared
//     memory, and one pass at the end adds the warps' partials of each output in a
//     fixed order; consecutive lanes store consecutive rows of a token.
// Experts that see few rows each are the same product over a table of code matrices (the expert loop,
// src/caif_device_moe_layer.cpp:534-557), up to 16 rows an entry (int8: 8), an expert of more being several entries: two CTAs of eight warps an SM, each with hundreds of weight rows; a round of
// tiles ends with its expert, and the next one's activations are awaited while the other CTA works.  Bound by the
// conversion and by the rounds' ends: 64 experts of 2048 x 1408 int4, 16 tokens top-6, three products 65 us (the
// streaming kernel 113, HBM 34).
// Codes and activations are exact in bf16 and products accumulate in fp32, so
// the result matches an fp32 GEMM on the dequantized weight up to summation
// order.  The summation order of an output does not depend on which CTA owns
// its row, so a row slice of a layer gives the same bits as the whole layer.
#include <atomic>
#include <mutex>
#include <vector>

#include "common.cuh"

namespace caifq
{

__device__ unsigned int g_decode_timeout_flag = 0;

// Reads and clears the flag (1 = some bounded wait ran out since the last call; -1 = query failed).
int take_decode_timeout_flag()
{
  unsigned int v = 0;
  const unsigned int zero = 0;
  if (cudaMemcpyFromSymbol(&v, g_decode_timeout_flag, sizeof(v)) != cudaSuccess)
  {
    return -1;
  }
  if (v != 0 && cudaMemcpyToSymbol(g_decode_timeout_flag, &zero, sizeof(zero)) != cudaSuccess)
  {
    return -1;
  }
  return v ? 1 : 0;
}

namespace
{

constexpr int kTileRows = 16;                    // weight rows per tile (the MMA's M)
constexpr int kRowQuantum = 8;                   // CTA row ranges start on multiples of this
constexpr uint32_t kSmemFull = 220u * 1024u;     // dynamic shared memory of a CTA that takes the SM alone
constexpr uint32_t kSmemHalf = 112u * 1024u;     // ... of one that leaves room for the next launch's CTA
constexpr uint32_t kSpinLimit = 1u << 22;        // polls of one wait before it gives up (tens of ms)
constexpr uint32_t kSpinLimitTest = 1u << 12;    // the same for the self-test of the give-up path

__device__ __forceinline__ uint32_t smem_u32(const void *p)
{
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count)
{
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes)
{
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}

__device__ __forceinline__ bool mbar_try(uint32_t addr, uint32_t parity)
{
  uint32_t done;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(done)
      : "r"(addr), "r"(parity)
      : "memory");
  return done != 0;
}

// Bounded wait: a copy that never lands turns into a flag and missing outputs instead of a hung GPU.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, uint32_t limit)
{
  const uint32_t addr = smem_u32(bar);
  for (uint32_t spin = 0; spin < limit; ++spin)
  {
    if (mbar_try(addr, parity))
    {
      return true;
    }
  }
  atomicExch(&g_decode_timeout_flag, 1u);
  return false;
}

__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void *src, uint32_t bytes, uint64_t *bar)
{
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

// D(16x8, fp32) = A(16x16, bf16, row) * B(16x8, bf16, col) + C.  Not volatile: a pure function of its operands, so
// the compiler may interleave independent accumulation chains.  C apart from D: a chain starts from values that
// are kept (or from zero) without copying them first.
__device__ __forceinline__ void mma_bf16_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                               uint32_t b0, uint32_t b1, const float *c)
{
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(c[0]), "f"(c[1]), "f"(c[2]), "f"(c[3]));
}

// 16 bytes of global memory into shared memory
__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src)
{
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }

template <int N>
__device__ __forceinline__ void cp_async_wait()
{
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// 32 bytes: a whole sector a lane (a lane's pieces of int4 codes have 64 bytes of x; every CTA reads all of x from L2, and
// that phase is 2 of a launch's 11 us: 4096 -> 4096, 16 tokens 8.8 -> 8.1 us, 14336 -> 4096 23.6 -> 21.9)
__device__ __forceinline__ void ldg256(const void *p, bool live, uint32_t *r)
{
  asm volatile(
      "{\n\t.reg .pred q;\n\t"
      "setp.ne.u32 q, %9, 0;\n\t"
      "mov.b32 %0, 0;\n\tmov.b32 %1, 0;\n\tmov.b32 %2, 0;\n\tmov.b32 %3, 0;\n\t"
      "mov.b32 %4, 0;\n\tmov.b32 %5, 0;\n\tmov.b32 %6, 0;\n\tmov.b32 %7, 0;\n\t"
      "@q ld.global.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n\t}"
      : "=&r"(r[0]), "=&r"(r[1]), "=&r"(r[2]), "=&r"(r[3]), "=&r"(r[4]), "=&r"(r[5]), "=&r"(r[6]), "=&r"(r[7])
      : "l"(p), "r"(live ? 1u : 0u)
      : "memory");
}

// activations are the previous kernel's output: never moved ahead of the wait on that kernel; zeros where not `live`
__device__ __forceinline__ void ldg128(const void *p, bool live, uint32_t &a, uint32_t &b, uint32_t &c, uint32_t &d)
{
  asm volatile(
      "{\n\t.reg .pred q;\n\t"
      "setp.ne.u32 q, %5, 0;\n\t"
      "mov.b32 %0, 0;\n\tmov.b32 %1, 0;\n\tmov.b32 %2, 0;\n\tmov.b32 %3, 0;\n\t"
      "@q ld.global.v4.u32 {%0,%1,%2,%3}, [%4];\n\t}"
      : "=&r"(a), "=&r"(b), "=&r"(c), "=&r"(d)
      : "l"(p), "r"(live ? 1u : 0u)
      : "memory");
}

__device__ __forceinline__ uint32_t sub_bf16x2(uint32_t a, uint32_t b)
{
  uint32_t d;
  asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}

__device__ __forceinline__ uint32_t lop3_and_or(uint32_t a, uint32_t b, uint32_t c)
{
  uint32_t d;
  asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(d) : "r"(a), "r"(b), "r"(c));  // (a & b) | c
  return d;
}

__device__ __forceinline__ uint32_t lop3_and_xor(uint32_t a, uint32_t b, uint32_t c)
{
  uint32_t d;
  asm("lop3.b32 %0, %1, %2, %3, 0x6A;" : "=r"(d) : "r"(a), "r"(b), "r"(c));  // (a & b) ^ c
  return d;
}

// Explicit shared-space accesses with 32-bit addresses.  Volatile keeps them in
// program order after the (volatile) wait that guards the data.
__device__ __forceinline__ uint4 lds128(uint32_t addr)
{
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
  return v;
}

__device__ __forceinline__ float lds_half(uint32_t addr)
{
  unsigned short h;
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(h) : "r"(addr));
  return __half2float(__ushort_as_half(h));
}

__device__ __forceinline__ float2 lds_f32x2(uint32_t addr)
{
  float2 v;
  asm volatile("ld.shared.v2.f32 {%0,%1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(addr));
  return v;
}

__device__ __forceinline__ void sts_f32x2(uint32_t addr, float a, float b)
{
  asm volatile("st.shared.v2.f32 [%0], {%1,%2};" ::"r"(addr), "f"(a), "f"(b) : "memory");
}


constexpr int kMaxSegments = 4;   // code matrices one launch may stream (layers that share their input)

struct DecodeParams
{
  // The rows of the launch are the rows of up to kMaxSegments code matrices laid end to end (q/k/v or
  // gate/up of one input): segment i covers rows seg_row0[i] .. seg_row0[i+1]; a single layer is one segment.
  const uint8_t *codes[kMaxSegments];   // [out_i, in] packed
  const void *scales[kMaxSegments];     // int4: fp16 per group; int8: fp32[1] or null
  int seg_row0[kMaxSegments + 1];
  int num_seg;
  const __nv_bfloat16 *x; // [m, in]
  void *y[kMaxPeers];     // [m, y_ld] on every GPU that receives the result (own buffer included)
  int num_y;
  int64_t y_ld;           // row pitch of the result, in elements
  int64_t y_col0;         // first column this launch writes
  int y_dtype;
  int accumulate;         // y = round_y(round_y(product) + y)
  int m;
  int in_dim;
  int out_dim;
  int groups_per_row;     // int4: in_dim / group_size
  int chunks_per_group;   // int4: group_size / 128
  int num_chunks;         // 64-byte pieces of a row
  int num_ksegs;          // passes over the CTA's rows, NCH pieces a warp each
  int num_quanta;         // ceil(out / 8)
  int tokp;               // tokens per parked row: m rounded up to 2, 4, 8 or 16
  int round_tiles;        // tiles whose partial sums fit the parking area: the CTA reduces and stores that often
  uint32_t scale_offset;  // byte offset of the scales in dynamic shared memory
  uint32_t scale_bytes;   // int4: one buffer of them (round_tiles tiles); two buffers when there are several rounds
  uint32_t park_offset;   // byte offset of the parked partial sums
  uint32_t row_bytes;     // packed bytes per weight row
  int entry_tiles;        // experts: tiles of one of them (out_dim: the rows of all of them)
  uint32_t spin_limit;    // polls of one wait before it gives up
  uint32_t stall_bytes;   // self-test only: bytes the first wait announces but never receives
};

// Experts: the same product for entries of one shape, each with its own codes and up to 16 rows of x.  Their weight rows
// lie end to end; out_dim is a multiple of 16, so a tile has one entry.
struct DecodeEntry
{
  const uint8_t *codes;
  const void *scales;
  void *c;               // [.., out_dim]; row 0 is packed row 0
  int row0;              // first packed row
  int rows;
};

constexpr int MAX_ENTRIES = 256;

template <int N>
struct DecodeTable
{
  DecodeEntry e[N];
};

// int4 codes are turned into the bf16 integers 24 + q (q in [-8,7]): the nibble, flipped to offset binary, is dropped
// into the upper mantissa bits of 16.0.  The constant is taken out again by starting each accumulator at -24 * (sum of x
// over the same 128 elements), so no subtract runs per weight.  The accumulator holds both for a while, so the constant
// sets the rounding: 136 + q (the nibble in the lower bits) saves a shift per eight weights, and was further from 64
// bits than an fp32 GEMM (4096 -> 4096, 5 tokens: 1.35e-6 against 7.4e-7; now 1.6e-7).
constexpr uint32_t kMinus24x2 = 0xC1C0C1C0u;

// WARPS: 8 or 16.  BITS: 4 or 8.  MT: token tiles of 8 (1 -> m <= 8, 2 -> m <= 16).
// NCH: chunks (64 bytes of one row: a quad of lanes x 16 bytes) per warp and pass; PCH of them per ring slot.
// Shared memory per CTA: the rings (8 KB a warp; 6 with two token tiles, whose parked sums take more), the
// scales, the parked sums.
template <int WARPS, int BITS, int MT, int NCH, int PCH>
struct DecodeCfg
{
  static constexpr int THREADS = WARPS * 32;
  static constexpr int CTAS_PER_SM = WARPS == 8 ? 2 : 1;
  // a multiple of the slots of a tile
  static constexpr int DEPTH = (MT == 2 && NCH / PCH == 1) ? 6 / PCH : 8 / PCH;
  static constexpr uint32_t SLOT_BYTES = PCH * 2u * 512u;
  static constexpr uint32_t WARP_RING = DEPTH * SLOT_BYTES;
};

// parked sums of one warp and tile: [16 rows][tokp], groups of four tokens of a row swapped so that the 16-byte
// reads of the reduction, eight rows at a time, fall into different banks
__device__ __forceinline__ uint32_t park_swizzle(int row, int tokp)
{
  return tokp == 16 ? static_cast<uint32_t>((row >> 1) & 3) : (tokp == 8 ? static_cast<uint32_t>((row >> 2) & 1) : 0u);
}

// An output as a plain fp32 sum of products: for tokens with an infinity or NaN, and where sums overflow only before the
// scale.  (Called without inlining it cost the 16-token forms 1.3 to 3 us a launch, registers being spilled around it.)
template <int BITS>
__device__ __forceinline__ float plain_sum(const DecodeParams &p, const uint8_t *codes, const void *scales, int row,
                                           const __nv_bfloat16 *x)
{
  codes += static_cast<size_t>(row) * p.row_bytes;
  const __half *group_scales = static_cast<const __half *>(scales) + static_cast<size_t>(row) * p.groups_per_row;
  const float tensor_scale = (BITS == 8 && scales != nullptr) ? *static_cast<const float *>(scales) : 1.0f;
  float sum = 0.0f;
#pragma unroll 1
  for (int k = 0; k < p.in_dim; ++k)
  {
    const int q = (BITS == 4) ? sign_extend_nibble((codes[k >> 1] >> (4 * (k & 1))) & 0xF) : static_cast<int8_t>(codes[k]);
    const float s = (BITS == 4) ? __half2float(group_scales[k / (128 * p.chunks_per_group)]) : tensor_scale;
    sum = fmaf(__fmul_rn(static_cast<float>(q), s), __bfloat162float(x[k]), sum);
  }
  return sum;
}

// N: entries of the table (experts), or 1: layers that share their input, which the parameters describe
template <int WARPS, int BITS, int MT, int NCH, int PCH, int N>
__global__ void __launch_bounds__(WARPS * 32, WARPS == 8 ? 2 : 1)
linear_decode_kernel(const __grid_constant__ DecodeParams p, const __grid_constant__ DecodeTable<N> table)
{
  constexpr bool EXPERTS = N > 1;
  constexpr int QUANTUM = EXPERTS ? kTileRows : kRowQuantum;
  typedef DecodeCfg<WARPS, BITS, MT, NCH, PCH> Cfg;
  constexpr int ELEMS = 128 / BITS;      // codes per 16-byte load: 32 or 16
  constexpr int CHUNK_K = 4 * ELEMS;     // k covered by a quad of lanes: 128 or 64
  constexpr int XR = ELEMS / 2;          // bf16x2 registers of x per chunk and token tile: 16 or 8
  constexpr int NSLAB = NCH / PCH;       // ring slots per tile and pass
  constexpr int CHAINS = (MT == 1) ? 2 : 1;   // accumulation chains per token tile
  static_assert(NCH % PCH == 0, "whole slots");

  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ uint64_t scale_bar[2];   // a round's scales have landed

  const int tid = threadIdx.x;
  const int warp = tid >> 5;
  const int lane = tid & 31;
  const int g = lane >> 2;  // A fragment rows g, g+8 (weight rows); B fragment column g (token)
  const int t = lane & 3;

  const int q_begin = static_cast<int>((static_cast<int64_t>(blockIdx.x) * p.num_quanta) / gridDim.x);
  const int q_end = static_cast<int>((static_cast<int64_t>(blockIdx.x + 1) * p.num_quanta) / gridDim.x);
  const int row_begin = q_begin * QUANTUM;
  const int row_end = min(q_end * QUANTUM, p.out_dim);
  const int my_tiles = (row_end - row_begin + kTileRows - 1) / kTileRows;
  const uint32_t smem_base = smem_u32(smem);
  const uint32_t ring = smem_base + static_cast<uint32_t>(warp) * Cfg::WARP_RING + static_cast<uint32_t>(lane) * 16u;

  // A code matrix and its rows' place among the launch's: of the entry of a tile, or of the layer that a row belongs to
  auto entry_of = [&](int tile) { return (q_begin + tile) / p.entry_tiles; };
  auto layer_of = [&](int row)
  {
    int sg = 0;
    while (sg + 1 < p.num_seg && row >= p.seg_row0[sg + 1])
    {
      ++sg;
    }
    return sg;
  };
  // The tiles are worked off in rounds, as many as the parking area takes; a round has one entry.
  auto round_stop = [&](int first)
  {
    int stop = min(first + p.round_tiles, my_tiles);
    if (EXPERTS)
    {
      stop = min(stop, (entry_of(first) + 1) * p.entry_tiles - q_begin);
    }
    return stop;
  };

  // The copies run DEPTH slots ahead of the compute loop, in its order: rounds, passes over k, tiles, slots.  Rows past
  // the CTA's last one are read as that one (their sums are never stored), pieces past the row's end not at all
  // (their activations are zero).
  int f_round = 0;   // first tile of the round being fetched
  // (one table entry: rounds are counted, not kept in a register: 512 -> 4096, 16 tokens 4.25 us, 4.50 kept)
  int f_stop = round_stop(0);
  int f_tile = 0;
  int f_kseg = 0;
  const uint8_t *f_lo;   // this lane's first piece of row g, and of row g + 8, of the tile
  const uint8_t *f_hi;
  auto row_ptr = [&](int row)
  {
    row = min(row, row_end - 1);
    const uint8_t *base = p.codes[0];
    if (EXPERTS)
    {
      const int entry = row / (p.entry_tiles * kTileRows);
      base = table.e[entry].codes;
      row -= entry * p.entry_tiles * kTileRows;
    }
    else if (p.num_seg > 1)
    {
      const int sg = layer_of(row);
      base = p.codes[sg];
      row -= p.seg_row0[sg];
    }
    return base + static_cast<size_t>(row) * p.row_bytes + static_cast<uint32_t>((f_kseg * NCH * WARPS + warp) * 64 + t * 16);
  };
  auto fetch_rows = [&]()
  {
    const int row = row_begin + f_tile * kTileRows + g;
    f_lo = row_ptr(row);
    f_hi = EXPERTS ? f_lo + 8u * p.row_bytes : row_ptr(row + 8);
  };
  auto fetch = [&](int slab, uint32_t dst)
  {
    if (f_round < my_tiles)
    {
      const int pieces = p.num_chunks - f_kseg * (NCH * WARPS) - warp;
#pragma unroll
      for (int j = 0; j < PCH; ++j)
      {
        const int off = (slab * PCH + j) * WARPS;
        if (off < pieces)
        {
          cp_async16(dst + j * 1024u, f_lo + off * 64);
          cp_async16(dst + j * 1024u + 512u, f_hi + off * 64);
        }
      }
      if (slab == NSLAB - 1)
      {
        if (++f_tile == (EXPERTS ? f_stop : min(f_round + p.round_tiles, my_tiles)))
        {
          if (++f_kseg == p.num_ksegs)
          {
            f_kseg = 0;
            f_round = f_tile;
            f_stop = f_round < my_tiles ? round_stop(f_round) : f_stop;
          }
          f_tile = f_round;
        }
        if (EXPERTS && f_tile > f_round)
        {
          f_lo += static_cast<uint32_t>(kTileRows) * p.row_bytes;
          f_hi += static_cast<uint32_t>(kTileRows) * p.row_bytes;
        }
        else
        {
          fetch_rows();
        }
      }
    }
    cp_async_commit();
  };
  // One thread copies a round's scales: contiguous in memory, one copy per code matrix the rows touch.
  auto fetch_scales = [&](int round, int first_tile)
  {
    uint64_t *bar = &scale_bar[round & 1];
    const int row0 = row_begin + first_tile * kTileRows;
    const int row1 = min(row_end, row_begin + round_stop(first_tile) * kTileRows);
    const uint32_t per_row = (BITS == 4) ? static_cast<uint32_t>(p.groups_per_row) * 2u : 0u;
    mbar_expect_tx(bar, static_cast<uint32_t>(row1 - row0) * per_row + (round == 0 ? p.stall_bytes : 0u));
    if (BITS == 4)
    {
      uint32_t dst = smem_base + p.scale_offset + static_cast<uint32_t>(round & 1) * p.scale_bytes;
      for (int row = row0; row < row1;)
      {
        const int sg = EXPERTS ? entry_of(first_tile) : layer_of(row);
        const int sg_row0 = EXPERTS ? sg * p.entry_tiles * kTileRows : p.seg_row0[sg];
        const int n = EXPERTS ? row1 - row : min(row1, p.seg_row0[sg + 1]) - row;
        const uint8_t *src = static_cast<const uint8_t *>(EXPERTS ? table.e[sg].scales : p.scales[sg]) +
                             static_cast<size_t>(row - sg_row0) * per_row;
        bulk_g2s(dst, src, static_cast<uint32_t>(n) * per_row, bar);
        dst += static_cast<uint32_t>(n) * per_row;
        row += n;
      }
    }
  };

  // The frozen codes and scales never depend on earlier work in the stream: their copies start before the wait on
  // the previous kernel.  The next kernel in the stream may place its CTAs as soon as this grid's CTAs have all
  // come this far (programmatic dependent launch).
  const int f_stop_0 = f_stop;
  fetch_rows();
#pragma unroll
  for (int i = 0; i < Cfg::DEPTH; ++i)
  {
    fetch(i % NSLAB, ring + static_cast<uint32_t>(i) * Cfg::SLOT_BYTES);
  }
  if (tid == 0)
  {
    mbar_init(&scale_bar[0], 1);
    mbar_init(&scale_bar[1], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fetch_scales(0, 0);
    if (f_stop_0 < my_tiles)
    {
      fetch_scales(1, f_stop_0);
    }
  }
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  // Activations and the output are touched only after the previous kernel has completed.
  asm volatile("griddepcontrol.wait;" ::: "memory");

  // Token fragments (B operand) of one pass over k.  For the 16 bytes of codes a lane reads, the register order
  // pairs the elements the way the logic-op dequantization emits them:
  //   int4, word wi: (8wi+0, 8wi+4) (8wi+2, 8wi+6) (8wi+1, 8wi+5) (8wi+3, 8wi+7)
  //   int8, word wi: (4wi+0, 4wi+2) (4wi+1, 4wi+3)
  uint32_t xf[NCH][MT][XR];
  float sx[NCH][MT][4];     // int4: -24 * (sum of x over the chunk's 128 elements) as an accumulator fragment
  uint32_t scale_off[NCH];  // byte offset of row g's scale for the chunk inside a tile's scales
  auto load_x = [&](int kseg, const __nv_bfloat16 *x, int m)
  {
    // all loads first: one round trip
    const bool wide = (reinterpret_cast<uintptr_t>(x) & 31u) == 0;   // (rows are a multiple of 128 bytes)
#pragma unroll
    for (int ch = 0; ch < NCH; ++ch)
    {
      const int c = (kseg * NCH + ch) * WARPS + warp;
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
      {
        const int token = g + 8 * mt;
        const bool live = c < p.num_chunks && token < m;
        const __nv_bfloat16 *src = x + static_cast<size_t>(token) * p.in_dim + c * CHUNK_K + t * ELEMS;
        if (wide)
        {
#pragma unroll
          for (int i = 0; i < XR / 8; ++i)
          {
            ldg256(src + 16 * i, live, &xf[ch][mt][8 * i]);
          }
        }
        else
        {
#pragma unroll
          for (int i = 0; i < XR / 4; ++i)
          {
            ldg128(src + 8 * i, live, xf[ch][mt][4 * i], xf[ch][mt][4 * i + 1], xf[ch][mt][4 * i + 2], xf[ch][mt][4 * i + 3]);
          }
        }
      }
    }
#pragma unroll
    for (int ch = 0; ch < NCH; ++ch)
    {
      const int c = (kseg * NCH + ch) * WARPS + warp;
      scale_off[ch] = (BITS == 4 && c < p.num_chunks)
                          ? static_cast<uint32_t>(g * p.groups_per_row + c / p.chunks_per_group) * 2u
                          : 0u;
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
      {
        uint32_t(&f)[XR] = xf[ch][mt];
#pragma unroll
        for (int wi = 0; wi < 4; ++wi)
        {
          if (BITS == 4)
          {
            const uint32_t r0 = f[(4 * wi + 0) % XR], r1 = f[(4 * wi + 1) % XR], r2 = f[(4 * wi + 2) % XR],
                           r3 = f[(4 * wi + 3) % XR];
            f[(4 * wi + 0) % XR] = __byte_perm(r0, r2, 0x5410);
            f[(4 * wi + 1) % XR] = __byte_perm(r1, r3, 0x5410);
            f[(4 * wi + 2) % XR] = __byte_perm(r0, r2, 0x7632);
            f[(4 * wi + 3) % XR] = __byte_perm(r1, r3, 0x7632);
          }
          else
          {
            const uint32_t r0 = f[2 * wi], r1 = f[2 * wi + 1];
            f[2 * wi] = __byte_perm(r0, r1, 0x5410);
            f[2 * wi + 1] = __byte_perm(r0, r1, 0x7632);
          }
        }
        // the sums come from the tensor core too: the accumulators of weight rows whose codes are all -24
        float c0[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        if (BITS == 4)
        {
          float c1[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
          for (int j = 0; j < XR / 2; j += 2)
          {
            mma_bf16_16816(c0, kMinus24x2, kMinus24x2, kMinus24x2, kMinus24x2, f[2 * j], f[2 * j + 1], c0);
            mma_bf16_16816(c1, kMinus24x2, kMinus24x2, kMinus24x2, kMinus24x2, f[2 * j + 2], f[2 * j + 3], c1);
          }
#pragma unroll
          for (int i = 0; i < 4; ++i)
          {
            c0[i] += c1[i];
          }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
        {
          sx[ch][mt][i] = c0[i];
        }
      }
    }
  };

  const uint32_t scale8_off = static_cast<uint32_t>(8 * p.groups_per_row) * 2u;
  const uint32_t tile_scale_bytes = 2u * scale8_off;
  const uint32_t park_warp_bytes = static_cast<uint32_t>(kTileRows * p.tokp) * 4u;
  const uint32_t park_tile_bytes = WARPS * park_warp_bytes;
  const uint32_t park_base = smem_base + p.park_offset;
  // a lane's two tokens of a row are one 8-byte store (row g + 8 has the swizzle of row g)
  uint32_t park_off[MT];
#pragma unroll
  for (int mt = 0; mt < MT; ++mt)
  {
    const uint32_t quad = static_cast<uint32_t>((t >> 1) + 2 * mt) ^ park_swizzle(g, p.tokp);
    park_off[mt] = static_cast<uint32_t>(warp) * park_warp_bytes +
                   (static_cast<uint32_t>(g * p.tokp) + 4u * quad + 2u * static_cast<uint32_t>(t & 1)) * 4u;
  }
  const float zero4[4] = {0.0f, 0.0f, 0.0f, 0.0f};
  uint32_t slot = 0;   // byte offset in the ring
  int round = 0;
  int entry = -1;
  for (int round_begin = 0, round_end = 0; round_begin < my_tiles; round_begin = round_end, ++round)
  {
    round_end = EXPERTS ? round_stop(round_begin) : min(round_begin + p.round_tiles, my_tiles);
    const int entry_before = entry;
    entry = EXPERTS ? entry_of(round_begin) : 0;
    const int m = EXPERTS ? table.e[entry].rows : p.m;
    const __nv_bfloat16 *x = p.x + (EXPERTS ? static_cast<size_t>(table.e[entry].row0) * p.in_dim : 0);
    const uint32_t scale_base = smem_base + p.scale_offset + static_cast<uint32_t>(round & 1) * p.scale_bytes;
    for (int kseg = 0; kseg < p.num_ksegs; ++kseg)
    {
      if ((EXPERTS ? entry != entry_before : round == 0) || p.num_ksegs > 1)
      {
        load_x(kseg, x, m);
      }
      if (kseg == 0)
      {
        if (round == 0)
        {
          __syncthreads();   // the barriers are initialised
        }
        const bool landed = mbar_wait(&scale_bar[round & 1], static_cast<uint32_t>(round >> 1) & 1u, p.spin_limit);
        if (__syncthreads_or(landed ? 0 : 1))
        {
          // A wait ran out; the outputs stay unwritten and the host sees the flag.  Copies that were started must
          // land before the shared memory belongs to another CTA.
          cp_async_wait<0>();
          for (int i = 0; i < 64; ++i)
          {
            __nanosleep(2000);
          }
          return;
        }
      }
      for (int tile = round_begin; tile < round_end; ++tile)
      {
        const uint32_t tile_scales = scale_base + static_cast<uint32_t>(tile - round_begin) * tile_scale_bytes;
        // yacc[mt][0..1]: row g, tokens 2t, 2t+1 of tile mt;  [2..3]: row g+8
        float yacc[MT][4];
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
        {
          yacc[mt][0] = yacc[mt][1] = yacc[mt][2] = yacc[mt][3] = 0.0f;
        }
#pragma unroll
        for (int slab = 0; slab < NSLAB; ++slab)
        {
          cp_async_wait<Cfg::DEPTH - 1>();
          const uint32_t src = ring + slot;
#pragma unroll
          for (int j = 0; j < PCH; ++j)
          {
            const int ch = slab * PCH + j;
            {
              const uint4 lo = lds128(src + j * 1024u);
              const uint4 hi = lds128(src + j * 1024u + 512u);
              const uint32_t wlo[4] = {lo.x, lo.y, lo.z, lo.w};
              const uint32_t whi[4] = {hi.x, hi.y, hi.z, hi.w};
              float s_lo = 0.0f;
              float s_hi = 0.0f;
              if (BITS == 4)
              {
                s_lo = lds_half(tile_scales + scale_off[ch]);
                s_hi = lds_half(tile_scales + scale_off[ch] + scale8_off);
              }
              float c[CHAINS][MT][4];
#pragma unroll
              for (int wi = 0; wi < 4; ++wi)
              {
                if (BITS == 4)
                {
                  uint32_t a_lo[4];
                  uint32_t a_hi[4];
                  {
                    const uint32_t ev = lop3_and_xor(wlo[wi] << 3, 0x78787878u, 0xC0C0C0C0u);
                    const uint32_t od = lop3_and_xor(wlo[wi] >> 1, 0x78787878u, 0xC0C0C0C0u);
                    a_lo[0] = __byte_perm(ev, 0x41414141u, 0x4240);
                    a_lo[1] = __byte_perm(ev, 0x41414141u, 0x4341);
                    a_lo[2] = __byte_perm(od, 0x41414141u, 0x4240);
                    a_lo[3] = __byte_perm(od, 0x41414141u, 0x4341);
                  }
                  {
                    const uint32_t ev = lop3_and_xor(whi[wi] << 3, 0x78787878u, 0xC0C0C0C0u);
                    const uint32_t od = lop3_and_xor(whi[wi] >> 1, 0x78787878u, 0xC0C0C0C0u);
                    a_hi[0] = __byte_perm(ev, 0x41414141u, 0x4240);
                    a_hi[1] = __byte_perm(ev, 0x41414141u, 0x4341);
                    a_hi[2] = __byte_perm(od, 0x41414141u, 0x4240);
                    a_hi[3] = __byte_perm(od, 0x41414141u, 0x4341);
                  }
#pragma unroll
                  for (int h = 0; h < 2; ++h)
                  {
                    const int jj = 2 * wi + h;  // k-step: pairs 2jj, 2jj+1
#pragma unroll
                    for (int mt = 0; mt < MT; ++mt)
                    {
                      mma_bf16_16816(c[h % CHAINS][mt], a_lo[2 * h], a_hi[2 * h], a_lo[2 * h + 1], a_hi[2 * h + 1],
                                     xf[ch][mt][2 * jj], xf[ch][mt][2 * jj + 1],
                                     jj == 0 ? sx[ch][mt] : (jj < CHAINS ? zero4 : c[h % CHAINS][mt]));
                    }
                  }
                }
                else
                {
                  uint32_t a_lo[2];
                  uint32_t a_hi[2];
#pragma unroll
                  for (int sh = 0; sh < 2; ++sh)
                  {
                    const uint32_t sel = sh ? 0x4341u : 0x4240u;
                    const uint32_t pl = __byte_perm(wlo[wi], 0u, sel);
                    const uint32_t ph = __byte_perm(whi[wi], 0u, sel);
                    a_lo[sh] =
                        sub_bf16x2(lop3_and_or(pl, 0x007F007Fu, 0x43004300u), lop3_and_or(pl, 0x00800080u, 0x43004300u));
                    a_hi[sh] =
                        sub_bf16x2(lop3_and_or(ph, 0x007F007Fu, 0x43004300u), lop3_and_or(ph, 0x00800080u, 0x43004300u));
                  }
#pragma unroll
                  for (int mt = 0; mt < MT; ++mt)
                  {
                    mma_bf16_16816(c[wi % CHAINS][mt], a_lo[0], a_hi[0], a_lo[1], a_hi[1], xf[ch][mt][2 * wi],
                                   xf[ch][mt][2 * wi + 1], wi < CHAINS ? zero4 : c[wi % CHAINS][mt]);
                  }
                }
              }
#pragma unroll
              for (int mt = 0; mt < MT; ++mt)
              {
                float sum[4];
#pragma unroll
                for (int i = 0; i < 4; ++i)
                {
                  sum[i] = (CHAINS == 2) ? (c[0][mt][i] + c[CHAINS - 1][mt][i]) : c[0][mt][i];
                }
                if (BITS == 4)
                {
                  // the chunk lies inside one scale group of rows g and g+8; scaling per
                  // 128-element chunk equals scaling per group up to rounding order
                  yacc[mt][0] = fmaf(s_lo, sum[0], yacc[mt][0]);
                  yacc[mt][1] = fmaf(s_lo, sum[1], yacc[mt][1]);
                  yacc[mt][2] = fmaf(s_hi, sum[2], yacc[mt][2]);
                  yacc[mt][3] = fmaf(s_hi, sum[3], yacc[mt][3]);
                }
                else
                {
#pragma unroll
                  for (int i = 0; i < 4; ++i)
                  {
                    yacc[mt][i] += sum[i];
                  }
                }
              }
            }
          }
          // the slot's contents are in registers (the MMAs above consumed them): refill it
          fetch(slab, src);
          slot = (slot + Cfg::SLOT_BYTES == Cfg::WARP_RING) ? 0u : slot + Cfg::SLOT_BYTES;
        }
        // park this warp's partial sums of the tile; nobody else reads them before the end of the round
        const uint32_t d0 = park_base + static_cast<uint32_t>(tile - round_begin) * park_tile_bytes;
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
        {
          if (MT == 2 || 2 * t < p.tokp)
          {
            const uint32_t d = d0 + park_off[mt];
            const uint32_t d8 = d + static_cast<uint32_t>(8 * p.tokp) * 4u;
            if (kseg > 0)
            {
              const float2 o = lds_f32x2(d);
              const float2 o8 = lds_f32x2(d8);
              yacc[mt][0] += o.x;
              yacc[mt][1] += o.y;
              yacc[mt][2] += o8.x;
              yacc[mt][3] += o8.y;
            }
            sts_f32x2(d, yacc[mt][0], yacc[mt][1]);    // row g,   tokens 2t, 2t+1
            sts_f32x2(d8, yacc[mt][2], yacc[mt][3]);   // row g+8
          }
        }
      }
    }
    __syncthreads();
    if (tid == 0 && round_end < my_tiles)
    {
      const int next = round_stop(round_end);
      if (next < my_tiles)
      {
        fetch_scales(round + 2, next);
      }
    }

    // Cross-warp reduction: an output is the sum of its warps' partial sums in warp order.  A thread takes up to
    // four tokens of one row; consecutive lanes take consecutive rows, so a token's stores are contiguous across
    // the warp.  With peers the plain stores travel over NVLink and are complete when the kernel is.
    const int rows = (round_end - round_begin) * kTileRows;
    const int live_rows = min(rows, row_end - row_begin - round_begin * kTileRows);
    const int quads = (m + 3) >> 2;
    for (int tq = tid >> 7; tq < quads; tq += (WARPS * 32) / 128)
    {
      for (int local = tid & 127; local < live_rows; local += 128)
      {
        const int r16 = local & 15;
        const uint32_t src = park_base + static_cast<uint32_t>(local >> 4) * park_tile_bytes +
                             (static_cast<uint32_t>(r16 * p.tokp) +
                              4u * (static_cast<uint32_t>(tq) ^ park_swizzle(r16, p.tokp))) * 4u;
        float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        if (p.tokp > 2)
        {
#pragma unroll
          for (int w = 0; w < WARPS; ++w)
          {
            const uint4 v = lds128(src + static_cast<uint32_t>(w) * park_warp_bytes);
            acc[0] += __uint_as_float(v.x);
            acc[1] += __uint_as_float(v.y);
            acc[2] += __uint_as_float(v.z);
            acc[3] += __uint_as_float(v.w);
          }
        }
        else
        {
#pragma unroll
          for (int w = 0; w < WARPS; ++w)
          {
            const float2 v = lds_f32x2(src + static_cast<uint32_t>(w) * park_warp_bytes);
            acc[0] += v.x;
            acc[1] += v.y;
          }
        }
        const int row = row_begin + round_begin * kTileRows + local;
        if (BITS == 8)
        {
          const void *scale = EXPERTS ? table.e[entry].scales : p.scales[layer_of(row)];
          const float tensor_scale = scale != nullptr ? __ldg(static_cast<const float *>(scale)) : 1.0f;
#pragma unroll
          for (int i = 0; i < 4; ++i)
          {
            acc[i] *= tensor_scale;
          }
        }
        const int live = min(4, m - 4 * tq);
        // (summed before the scale, and int4 with an offset that turns an infinity into infinity - infinity)
        if (__builtin_expect(!(fabsf(acc[0]) + fabsf(acc[1]) + fabsf(acc[2]) + fabsf(acc[3]) <= 3.402823466e38f), 0))
        {
#pragma unroll 1
          for (int i = 0; i < live; ++i)
          {
            const float sum = i == 0 ? acc[0] : (i == 1 ? acc[1] : (i == 2 ? acc[2] : acc[3]));
            if (fabsf(sum) <= 3.402823466e38f)
            {
              continue;
            }
            const int sg = EXPERTS ? entry : layer_of(row);
            const int row0 = EXPERTS ? entry * p.entry_tiles * kTileRows : p.seg_row0[sg];
            const float v = plain_sum<BITS>(p, EXPERTS ? table.e[sg].codes : p.codes[sg],
                                            EXPERTS ? table.e[sg].scales : p.scales[sg], row - row0,
                                            x + static_cast<size_t>(4 * tq + i) * p.in_dim);
            acc[0] = i == 0 ? v : acc[0];
            acc[1] = i == 1 ? v : acc[1];
            acc[2] = i == 2 ? v : acc[2];
            acc[3] = i == 3 ? v : acc[3];
          }
        }
        int64_t idx = static_cast<int64_t>(4 * tq) * p.y_ld + p.y_col0 + row;
        if (EXPERTS)
        {
          idx = (static_cast<int64_t>(table.e[entry].row0) + 4 * tq) * p.y_ld + row - entry * p.entry_tiles * kTileRows;
#pragma unroll 1
          for (int i = 0; i < live; ++i, idx += p.y_ld)
          {
            store_from_float(table.e[entry].c, idx, p.y_dtype, i == 0 ? acc[0] : (i == 1 ? acc[1] : (i == 2 ? acc[2] : acc[3])));
          }
        }
        else if (p.y_dtype == CAIFQ_F32 && !p.accumulate && p.num_y == 1)
        {
          float *dst = static_cast<float *>(p.y[0]) + idx;
#pragma unroll
          for (int i = 0; i < 4; ++i, dst += p.y_ld)
          {
            if (i < live)
            {
              *dst = acc[i];
            }
          }
        }
        else
        {
#pragma unroll 1
          for (int i = 0; i < live; ++i, idx += p.y_ld)
          {
            float v = i == 0 ? acc[0] : (i == 1 ? acc[1] : (i == 2 ? acc[2] : acc[3]));
            if (p.accumulate)
            {
              v = round_through_rt(v, p.y_dtype) + load_as_float(p.y[0], idx, p.y_dtype);
            }
            for (int r = 0; r < p.num_y; ++r)
            {
              store_from_float(p.y[r], idx, p.y_dtype, v);
            }
          }
        }
      }
    }
    if (round_end < my_tiles)
    {
      __syncthreads();   // the parking area is free for the next round
    }
  }  // rounds
}

// One CTA per SM, fewer when the host runs a collective beside this kernel and wants to leave it SMs.  Experts take two, of
// half an SM each, and are not taken under a limit of either persistent kernel: twice as many CTAs would not keep to it, and
// with as many as it says half of each SM idles (three products of 64 experts of 2048 x 1408, 8 rows each, limit of 132:
// int4 176 us, int8 231, the streaming kernel 154 and 147).
int sm_count() { return persistent_ctas("CAIFQ_DECODE_CTAS"); }
int expert_ctas() { return 2 * device_sm_count(); }
bool limited()
{
  const int sms = device_sm_count();
  return persistent_ctas("CAIFQ_DECODE_CTAS") < sms || persistent_ctas("CAIFQ_UMMA_CTAS") < sms;
}

// Streams (per device) on which one of this library's calls has just written codes or scales.
std::mutex g_written_mutex;
std::vector<std::pair<int, cudaStream_t>> g_written;

thread_local bool t_stall_next = false;

}  // namespace

void note_codes_written(cudaStream_t s)
{
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lock(g_written_mutex);
  for (const auto &e : g_written)
  {
    if (e.first == dev && e.second == s)
    {
      return;
    }
  }
  g_written.emplace_back(dev, s);
}

bool take_codes_written(cudaStream_t s)
{
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lock(g_written_mutex);
  for (size_t i = 0; i < g_written.size(); ++i)
  {
    if (g_written[i].first == dev && g_written[i].second == s)
    {
      g_written.erase(g_written.begin() + static_cast<std::ptrdiff_t>(i));
      return true;
    }
  }
  return false;
}

void decode_stall_next_launch() { t_stall_next = true; }


namespace
{

template <int WARPS, int BITS, int MT, int NCH, int PCH, int N>
int launch_decode_inst(const DecodeParams &p, const DecodeTable<N> &table, uint32_t smem, cudaStream_t s)
{
  auto kernel = linear_decode_kernel<WARPS, BITS, MT, NCH, PCH, N>;
  static std::atomic<bool> configured[kMaxDevices];
  int dev = 0;
  CAIFQ_CHECK_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices)
  {
    set_error("frozen linear (decode): device ordinal %d out of range", dev);
    return CAIFQ_ERR_UNSUPPORTED;
  }
  if (!configured[dev].load(std::memory_order_acquire))
  {
    CAIFQ_CHECK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          static_cast<int>(kSmemFull)));
    configured[dev].store(true, std::memory_order_release);
  }
  int grid = N > 1 ? expert_ctas() : sm_count();
  if (grid > p.num_quanta)
  {
    grid = p.num_quanta;
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>(grid));
  cfg.blockDim = dim3(WARPS * 32);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  // codes written just ahead in this stream by one of the library's own calls: a plain launch
  // orders the early copies behind that kernel
  cfg.numAttrs = (dependent_launches() && !take_codes_written(s)) ? 1 : 0;
  CAIFQ_CHECK_CUDA(cudaLaunchKernelEx(&cfg, kernel, p, table));
  CAIFQ_CHECK_LAUNCH();
  return CAIFQ_OK;
}

int tokp_for(int64_t m) { return m <= 2 ? 2 : (m <= 4 ? 4 : (m <= 8 ? 8 : 16)); }

// How a launch is cut, by the shape of its rows and the most tokens of an entry.
struct Layout
{
  int warps;
  int nch;
  uint32_t scale_offset;
  uint32_t scale_bytes;
  uint32_t park_offset;
  uint32_t smem_bytes;   // 0: a tile does not fit
  int round_tiles;
};

// (w.out_dim: all the rows of the launch)
Layout layout_for(const caifq_weight &w, int64_t m, bool experts)
{
  Layout l{};
  const bool i4 = (w.storage == CAIFQ_I4);
  const int mt = (m > 8) ? 2 : 1;
  const int num_chunks = w.in_dim / (i4 ? 128 : 64);
  // Short rows (up to 1 KB of codes) keep few warps busy and their launches are short: eight warps on half an SM,
  // so that the next launch's CTA sits beside this one with its copies done (1024 -> 1024, m = 1: 2.4 us a launch
  // against 2.7).  Longer rows, and two token tiles, want the 16 warps: the launch is bound by the dequantization's
  // instructions and their latencies, not by its start (4096 -> 14336, m = 1: 10.4 us, 11.4 with eight, 11.6 with 32).
  // Experts: a CTA has hundreds of rows, and one of two on an SM works while the other waits for its next entry's activations.
  l.warps = (experts || (num_chunks <= 16 && mt == 1)) ? 8 : 16;
  // Chunks a warp holds token fragments of at a time: as many as 64 registers take (a lane needs 16 of them per
  // int4 chunk and token tile, 8 per int8 chunk), no more than the row has.
  const int most = (i4 ? 4 : 8) / mt;
  l.nch = experts ? 2 : 1;
  while (l.nch < most && l.nch * l.warps < num_chunks)
  {
    l.nch *= 2;
  }
  const bool deep = !(mt == 2 && l.nch <= 2);
  const uint32_t ring = static_cast<uint32_t>(l.warps) * (deep ? 8u : 6u) * 1024u;   // WARPS * DecodeCfg::WARP_RING
  const uint32_t scales = i4 ? static_cast<uint32_t>(kTileRows * (w.in_dim / w.group_size) * 2) : 0u;
  const uint32_t park = static_cast<uint32_t>(l.warps * kTileRows * tokp_for(m) * sizeof(float));
  const int quantum = experts ? kTileRows : kRowQuantum;
  const int quanta = (w.out_dim + quantum - 1) / quantum;
  int grid = experts ? expert_ctas() : sm_count();
  if (grid > quanta)
  {
    grid = quanta;
  }
  const int max_quanta = (quanta + grid - 1) / grid;
  const int max_tiles = (max_quanta * quantum + kTileRows - 1) / kTileRows;
  // all of a CTA's tiles in one round if they fit, else in several equal rounds
  const uint32_t budget = l.warps == 8 ? kSmemHalf : kSmemFull;
  auto align128 = [](uint32_t v) { return (v + 127u) & ~127u; };
  auto bytes = [&](int tiles, int buffers)
  { return ring + static_cast<uint32_t>(buffers) * align128(static_cast<uint32_t>(tiles) * scales) +
           static_cast<uint32_t>(tiles) * park; };
  int rounds = 1;
  int tiles = max_tiles;
  while (tiles > 1 && bytes(tiles, rounds > 1 || experts ? 2 : 1) > budget)
  {
    ++rounds;
    tiles = (max_tiles + rounds - 1) / rounds;
  }
  const int buffers = (tiles < max_tiles || experts) ? 2 : 1;   // (experts: a round ends with its entry, too)
  if (bytes(tiles, buffers) > kSmemFull)
  {
    return l;
  }
  l.round_tiles = tiles;
  l.scale_offset = ring;
  l.scale_bytes = align128(static_cast<uint32_t>(tiles) * scales);
  l.park_offset = ring + static_cast<uint32_t>(buffers) * l.scale_bytes;
  l.smem_bytes = bytes(tiles, buffers);
  return l;
}

}  // namespace

// int4 with groups of whole 128-element pieces, int8 with one scale or none.  bf16 compute in the reference rounds
// scale*code to bf16 before the product; this kernel keeps the exact fp32 scale.  Both are inside the bf16 tolerance, and
// fp32 compute is matched exactly.
static bool decode_weight(const caifq_weight &w)
{
  if (w.storage == CAIFQ_I4)
  {
    return w.scales != nullptr && w.group_size >= 128 && (w.group_size % 128) == 0 && (w.in_dim % w.group_size) == 0;
  }
  return w.storage == CAIFQ_I8 && (w.scales == nullptr || w.scheme == CAIFQ_PER_TENSOR) && (w.in_dim % 64) == 0;
}

// The launch's rows: the layer's own, or those of all the layers that share the input laid end to end.
static caifq_weight all_rows(const LinearArgs &args)
{
  caifq_weight w = args.w;
  for (int i = 0; i < args.num_more; ++i)
  {
    w.out_dim += args.more[i].out_dim;
  }
  return w;
}

bool decode_supported(const LinearArgs &args)
{
  if (args.num_more < 0 || args.num_more >= kMaxSegments || (args.num_more > 0 && args.more == nullptr))
  {
    return false;
  }
  for (int i = 0; i < args.num_more; ++i)
  {
    // layers of one launch have one storage, row length, scale rule; every one but the last ends on a
    // multiple of 8 rows, so that every copy of a straddling item stays a multiple of 16 bytes
    const caifq_weight &o = args.more[i];
    const caifq_weight &prev = (i == 0) ? args.w : args.more[i - 1];
    if (o.storage != args.w.storage || o.in_dim != args.w.in_dim || o.scheme != args.w.scheme ||
        o.group_size != args.w.group_size || (o.scales == nullptr) != (args.w.scales == nullptr) ||
        (prev.out_dim % kRowQuantum) != 0 || o.out_dim < 1 || (reinterpret_cast<uintptr_t>(o.codes) & 15u) != 0 ||
        (reinterpret_cast<uintptr_t>(o.scales) & 15u) != 0)
    {
      return false;
    }
  }
  const caifq_weight w = all_rows(args);
  const int x_dtype = args.a_dtype;
  const int64_t m = args.m;
  const int y_dtype = args.c_dtype;
  const int compute_dtype = args.compute_dtype;
  if (args.backward || args.a_prescale != 1.0f || (args.accumulate && args.num_peers > 0))
  {
    return false;
  }
  if (m < 1 || m > 16 || x_dtype != CAIFQ_BF16 || !is_float_dtype(y_dtype))
  {
    return false;
  }
  // Operands are exact in bf16 and accumulate in fp32: valid for fp32 and bf16
  // compute.  fp16 compute rounds x differently and goes elsewhere.
  if (compute_dtype != CAIFQ_F32 && compute_dtype != CAIFQ_BF16)
  {
    return false;
  }
  if (!decode_weight(w) || (w.storage == CAIFQ_I4 && (w.out_dim % kRowQuantum) != 0 && ((w.in_dim / w.group_size) % 8) != 0))
  {
    // (a ragged last item copies rows * groups_per_row fp16 scales: that is kept a multiple of 16 bytes)
    return false;
  }
  // a tile's scales and parked sums must fit beside the rings
  if (layout_for(w, m, false).smem_bytes == 0)
  {
    return false;
  }
  // bulk copies and 16-byte loads need aligned operands; a misaligned call goes to another kernel
  if ((reinterpret_cast<uintptr_t>(w.codes) & 15u) != 0 || (reinterpret_cast<uintptr_t>(w.scales) & 15u) != 0 ||
      (reinterpret_cast<uintptr_t>(args.a) & 15u) != 0)
  {
    return false;
  }
  return true;
}

static void shape_params(DecodeParams &p, const caifq_weight &w, const Layout &lay)
{
  const bool i4 = (w.storage == CAIFQ_I4);
  p.in_dim = w.in_dim;
  p.row_bytes = static_cast<uint32_t>(i4 ? w.in_dim / 2 : w.in_dim);
  p.groups_per_row = i4 ? w.in_dim / w.group_size : 0;
  p.chunks_per_group = i4 ? w.group_size / 128 : 1;
  p.num_chunks = w.in_dim / (i4 ? 128 : 64);
  p.num_ksegs = (p.num_chunks + lay.nch * lay.warps - 1) / (lay.nch * lay.warps);
  p.round_tiles = lay.round_tiles;
  p.scale_offset = lay.scale_offset;
  p.scale_bytes = lay.scale_bytes;
  p.park_offset = lay.park_offset;
}

int launch_linear_decode(const LinearArgs &args, cudaStream_t s)
{
  const caifq_weight w = all_rows(args);
  const int64_t m = args.m;
  const int y_dtype = args.c_dtype;
  DecodeParams p{};
  p.num_seg = 1 + args.num_more;
  p.seg_row0[0] = 0;
  for (int i = 0; i < p.num_seg; ++i)
  {
    const caifq_weight &seg = (i == 0) ? args.w : args.more[i - 1];
    p.codes[i] = static_cast<const uint8_t *>(seg.codes);
    p.scales[i] = seg.scales;
    p.seg_row0[i + 1] = p.seg_row0[i] + seg.out_dim;
  }
  for (int i = p.num_seg; i < kMaxSegments; ++i)
  {
    p.codes[i] = nullptr;
    p.scales[i] = nullptr;
    p.seg_row0[i + 1] = p.seg_row0[p.num_seg];
  }
  p.x = static_cast<const __nv_bfloat16 *>(args.a);
  if (args.num_peers > 0)
  {
    if (args.num_peers > kMaxPeers || args.c_peers == nullptr)
    {
      set_error("frozen linear (decode): at most %d peers", kMaxPeers);
      return CAIFQ_ERR_INVALID;
    }
    for (int r = 0; r < args.num_peers; ++r)
    {
      if (args.c_peers[r] == nullptr)
      {
        set_error("frozen linear (decode): null peer buffer %d", r);
        return CAIFQ_ERR_INVALID;
      }
      p.y[r] = args.c_peers[r];
    }
    p.num_y = args.num_peers;
    p.y_ld = args.c_ld;
    p.y_col0 = args.c_col0;
  }
  else
  {
    p.y[0] = args.c;
    p.num_y = 1;
    p.y_ld = w.out_dim;
    p.y_col0 = 0;
  }
  p.y_dtype = y_dtype;
  p.accumulate = args.accumulate ? 1 : 0;
  p.m = static_cast<int>(m);
  p.tokp = tokp_for(m);
  p.out_dim = w.out_dim;
  p.num_quanta = (w.out_dim + kRowQuantum - 1) / kRowQuantum;
  const Layout lay = layout_for(w, m, false);
  if (lay.smem_bytes == 0)
  {
    set_error("frozen linear (decode): row too long for the shared memory");
    return CAIFQ_ERR_UNSUPPORTED;
  }
  shape_params(p, w, lay);
  p.spin_limit = kSpinLimit;
  p.stall_bytes = 0;
  if (t_stall_next)
  {
    // self-test of the give-up path: the scales' wait announces 16 bytes that never arrive
    t_stall_next = false;
    p.spin_limit = kSpinLimitTest;
    p.stall_bytes = 16;
  }

  const bool i4 = w.storage == CAIFQ_I4;
  const int mt = (m > 8) ? 2 : 1;
  const DecodeTable<1> none{};
#define CAIFQ_DECODE_CASE(W, B, M, N)                                                      \
  if (lay.warps == W && lay.nch == N && mt == M)                                           \
  {                                                                                        \
    return launch_decode_inst<W, B, M, N, (N > 1 ? 2 : 1), 1>(p, none, lay.smem_bytes, s); \
  }
  if (i4)
  {
    CAIFQ_DECODE_CASE(8, 4, 1, 1)
    CAIFQ_DECODE_CASE(8, 4, 1, 2)
    CAIFQ_DECODE_CASE(16, 4, 1, 2)
    CAIFQ_DECODE_CASE(16, 4, 1, 4)
    CAIFQ_DECODE_CASE(16, 4, 2, 1)
    CAIFQ_DECODE_CASE(16, 4, 2, 2)
  }
  else
  {
    CAIFQ_DECODE_CASE(8, 8, 1, 1)
    CAIFQ_DECODE_CASE(8, 8, 1, 2)
    CAIFQ_DECODE_CASE(16, 8, 1, 2)
    CAIFQ_DECODE_CASE(16, 8, 1, 4)
    CAIFQ_DECODE_CASE(16, 8, 1, 8)
    CAIFQ_DECODE_CASE(16, 8, 2, 1)
    CAIFQ_DECODE_CASE(16, 8, 2, 2)
    CAIFQ_DECODE_CASE(16, 8, 2, 4)
  }
#undef CAIFQ_DECODE_CASE
  set_error("frozen linear (decode): no kernel instance for in_dim=%d m=%lld", w.in_dim, static_cast<long long>(m));
  return CAIFQ_ERR_UNSUPPORTED;
}

// Experts: entries of more than 16 rows are taken 16 at a time (their codes come from L2 again).
static int decode_entries(const GroupedStreamArgs &g, DecodeTable<MAX_ENTRIES> *table, int &most)
{
  int count = 0;
  most = 0;
  for (int e = 0; e < g.count; ++e)
  {
    for (int row = g.row_begin[e]; row < g.row_end[e]; row += 16)
    {
      const int rows = g.row_end[e] - row < 16 ? g.row_end[e] - row : 16;
      if (count == MAX_ENTRIES)
      {
        return -1;
      }
      if (table != nullptr)
      {
        table->e[count] = DecodeEntry{static_cast<const uint8_t *>(g.weights[e].codes), g.weights[e].scales, g.c[e], row, rows};
      }
      most = rows > most ? rows : most;
      ++count;
    }
  }
  return count;
}

bool decode_grouped_supported(const GroupedStreamArgs &g)
{
  int most = 0;
  const int entries = g.count < 1 ? -1 : decode_entries(g, nullptr, most);
  if (limited() || entries < 1 || g.accumulate || !is_float_dtype(g.c_dtype) || (reinterpret_cast<uintptr_t>(g.a) & 15u) != 0 ||
      (g.compute_dtype != CAIFQ_F32 && g.compute_dtype != CAIFQ_BF16))
  {
    return false;
  }
  const caifq_weight &w0 = g.weights[0];
  if (w0.storage != CAIFQ_I4 && most > 8)   // (a second tile of tokens pays for int4 alone, see the caller)
  {
    return false;
  }
  if ((w0.out_dim % kTileRows) != 0 || static_cast<int64_t>(entries) * w0.out_dim > 0x7FFFFFFF)
  {
    return false;
  }
  for (int e = 0; e < g.count; ++e)
  {
    const caifq_weight &w = g.weights[e];
    if (!decode_weight(w) || w.storage != w0.storage || w.in_dim != w0.in_dim || w.out_dim != w0.out_dim ||
        w.group_size != w0.group_size || (reinterpret_cast<uintptr_t>(w.codes) & 15u) != 0 ||
        (w.storage == CAIFQ_I4 && (reinterpret_cast<uintptr_t>(w.scales) & 15u) != 0))
    {
      return false;
    }
  }
  caifq_weight all = w0;
  all.out_dim *= entries;
  return layout_for(all, most, true).smem_bytes != 0;
}

int launch_linear_decode_grouped(const GroupedStreamArgs &g, cudaStream_t s)
{
  static thread_local DecodeTable<MAX_ENTRIES> table;
  int most = 0;
  const int entries = decode_entries(g, &table, most);
  if (entries < 1)
  {
    return entries == 0 ? CAIFQ_OK : CAIFQ_ERR_UNSUPPORTED;
  }
  caifq_weight w = g.weights[0];
  DecodeParams p{};
  p.entry_tiles = w.out_dim / kTileRows;
  p.y_ld = w.out_dim;
  w.out_dim *= entries;
  const Layout lay = layout_for(w, most, true);
  if (lay.smem_bytes == 0)
  {
    set_error("frozen experts (decode): row too long for the shared memory");
    return CAIFQ_ERR_UNSUPPORTED;
  }
  shape_params(p, w, lay);
  p.num_seg = 1;
  p.x = static_cast<const __nv_bfloat16 *>(g.a);
  p.num_y = 1;
  p.y_dtype = g.c_dtype;
  p.m = most;
  p.tokp = tokp_for(most);
  p.out_dim = w.out_dim;
  p.num_quanta = w.out_dim / kTileRows;
  p.spin_limit = kSpinLimit;
  const int mt = (most > 8) ? 2 : 1;
#define CAIFQ_DECODE_CASE(B, M, N)                                                                         \
  if (mt == M && lay.nch == N)                                                                             \
  {                                                                                                        \
    return launch_decode_inst<8, B, M, N, 2, MAX_ENTRIES>(p, table, lay.smem_bytes, s);                    \
  }
  if (w.storage == CAIFQ_I4)
  {
    CAIFQ_DECODE_CASE(4, 1, 2)
    CAIFQ_DECODE_CASE(4, 1, 4)
    CAIFQ_DECODE_CASE(4, 2, 2)
  }
  else
  {
    CAIFQ_DECODE_CASE(8, 1, 2)
    CAIFQ_DECODE_CASE(8, 1, 4)
    CAIFQ_DECODE_CASE(8, 1, 8)
  }
#undef CAIFQ_DECODE_CASE
  set_error("frozen experts (decode): no kernel instance for in_dim=%d rows=%d", w.in_dim, most);
  return CAIFQ_ERR_UNSUPPORTED;
}

}  // namespace caifq
