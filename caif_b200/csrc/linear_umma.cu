// Tensor-core frozen-linear GEMM for many tokens (prefill / training shapes):
//
//   forward : C[m, out] = A[m, in]  . W_deq[out, in]^T     (ForwardImpl,  src/caif_device_frozen_linear.cpp:381-524)
//   backward: C[m, in]  = A[m, out] . W_deq[out, in]       (BackwardImpl, src/caif_device_frozen_linear.cpp:526-660)
//
// Blackwell-native: tcgen05.mma (kind::f16, bf16 operands, fp32 accumulators in
// TMEM), operands staged in shared memory in the canonical 128-byte-swizzled
// layouts, activations fed by TMA.  The weight never exists as a float matrix
// in memory (the reference dequantizes [out,in] to fp32 and hands it to cuBLAS,
// :288-378): eight warps read the packed codes straight from global memory,
// expand them to bf16 in registers and write the B operand tile into shared
// memory, one k-block ahead of the MMA warp.
//
// One persistent CTA per SM, 14 warps:
//   warp 0      TMA producer for the activation tiles (warp 10 for the weight tiles
//               when the weight is already bf16)
//   warp 1      TMEM allocation, MMA issue (one elected lane)
//   warps 2-5   epilogue: TMEM -> registers -> scale -> global
//   warps 6-13  dequantization of the weight tile
// A bf16 weight has no dequantization: warp 10 copies its tiles and warps 6-9 join
// the epilogue.
// Tiles of 256 rows x 128 or 256 columns x 64 k (a single CTA: two 128-row MMAs that
// share a weight tile), or 256 rows on a CTA pair (a bf16 weight: 64 to 256 columns in
// steps of 32), three to six pipeline stages; two accumulator sets in TMEM, so that the
// epilogue of one tile overlaps the main loop of the next, except for a single CTA's
// 256-wide tile, which fills TMEM.
//
// Forward uses the weight tile K-major (k = in is contiguous in memory);
// backward uses the SAME codes MN-major (n = in is contiguous), so dX needs no
// transposed copy of the weight.
//
// Exactness: int8 codes are exact in bf16 and the per-tensor scale multiplies
// the fp32 accumulator in the epilogue, so with bf16 activations the products
// are exact and the result matches an fp32 GEMM up to summation order.  int4
// weights converted here are code * bf16(scale), rounded to bf16 (fp32 compute: two
// bf16 terms of scale * code); one that was expanded before the launch is a bf16 weight
// of bf16(scale * code), the operand the reference's bf16 compute cell builds
// (dequantize to fp32, then To(bf16)).
//
// Every wait is bounded; a wait that runs out sets a flag that the host can
// read and lets the kernel finish (with wrong numbers) instead of hanging.
#include <cstdlib>

#include <atomic>

#include "umma.cuh"

namespace caifq
{

__device__ unsigned int g_umma_timeout_flag = 0;

namespace
{
thread_local bool t_umma_stall_next = false;
}

// self-test hook: the next single-layer tensor-core launch of this thread waits for bytes that never arrive
void umma_stall_next_launch() { t_umma_stall_next = true; }

bool take_umma_stall()
{
  const bool stall = t_umma_stall_next;
  t_umma_stall_next = false;
  return stall;
}

// Reads and clears the flag (1 = some bounded wait ran out since the last call; -1 = query failed).
int take_umma_timeout_flag()
{
  unsigned int v = 0;
  const unsigned int zero = 0;
  if (cudaMemcpyFromSymbol(&v, g_umma_timeout_flag, sizeof(v)) != cudaSuccess)
  {
    return -1;
  }
  if (v != 0 && cudaMemcpyToSymbol(g_umma_timeout_flag, &zero, sizeof(zero)) != cudaSuccess)
  {
    return -1;
  }
  return v ? 1 : 0;
}

namespace
{

constexpr int BM_SUB = 128;          // rows of one MMA
constexpr int MT = 2;                // MMAs (row sub-tiles) per weight tile
constexpr int BM = BM_SUB * MT;      // 256
// BN (columns of the output tile, N of one MMA) is a template parameter: 128 or 256
constexpr int kBand = 8;             // row tiles of a band of the schedule
constexpr int BK = 64;               // one 128-byte swizzle span of bf16
constexpr int UMMA_K = 16;
constexpr int A_SUB_BYTES = BM_SUB * BK * 2;       // 16 KB

constexpr int MAX_STAGES = 6;
constexpr int TMEM_COLS = 512;
constexpr int NUM_WARPS = 14;
constexpr int NUM_THREADS = NUM_WARPS * 32;
constexpr int DEQ_WARP0 = 6;
constexpr int DEQ_THREADS = 8 * 32;
constexpr int B_WARP = 10;           // bf16 weights: the warp that copies their tiles
// Teams of dequant warps (see the dequantization role): two for a single CTA's tile; four for a CTA pair,
// whose k-blocks take half as long while a conversion's latency chain (wait, loads, ~150 instructions,
// stores, proxy fence, arrive) stays the same (two teams: 750-830 TFLOP/s on 4096 x 4096 int8, four: 980-1150).
__host__ __device__ constexpr int deq_teams(bool pair) { return pair ? 4 : 2; }

// A weight tile (BM = 256 activation rows x BN output columns) is worked on by one CTA, as two 128-row MMAs that
// share the staged weights, or -- PAIR -- by the two CTAs of a cluster with one `cta_group::2` MMA of 256 rows:
// each CTA stages its own 128 activation rows and its own half of the weight rows, so an SM moves half the
// operand bytes through its shared memory per flop and the 256 accumulator columns leave room for a second
// accumulator set (the epilogue overlaps the next tile).
template <int BN, int PLANES = 1, bool PAIR = false>
struct TileCfg
{
  static constexpr int MTK = PAIR ? 1 : MT;                       // 128-row sub-tiles of a CTA
  static constexpr int BNC = PAIR ? BN / 2 : BN;                  // weight-tile rows a CTA stages
  static constexpr int A_BYTES = A_SUB_BYTES * MTK;               // 16 or 32 KB
  static constexpr int B_PLANE_BYTES = BNC * BK * 2;              // 16 or 32 KB
  static constexpr int B_STAGE_BYTES = B_PLANE_BYTES * PLANES;
  static constexpr int STAGE_BYTES = A_BYTES + B_STAGE_BYTES;
  static constexpr int STAGES = (192 * 1024) / STAGE_BYTES;       // 192 KB of operands in every case: 3, 4 or 6
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024;  // + slack to align the base to 1024
  static constexpr int ACC_COLS = PAIR ? BN : MT * BN;            // accumulator columns of a CTA per tile
  static constexpr int ACC_BUFS = TMEM_COLS / ACC_COLS;           // 2 (epilogue overlaps the next tile) or 1
  static_assert(!PAIR || BN == 256, "tile pairs are 256 columns wide");
  static_assert(STAGES >= 3 && STAGES <= MAX_STAGES, "operand ring depth");
};

struct UmmaParams
{
  const uint8_t *codes;
  const void *scales;
  void *c;
  int c_dtype;
  int accumulate;    // epilogue: c = round_c(round_c(acc) + c_old)
  int64_t m;
  int n_total;       // columns of C
  int k_total;       // reduction length
  int in_dim;        // row length of the code matrix
  int group_size;    // int4
  int groups_per_row;  // int4: in_dim / group_size
  int num_m_tiles;
  int num_n_tiles;
  int band;            // row tiles of a band of the schedule (see locate_tile)
  int wide_stores;     // outputs (and what the SwiGLU backward reads) are 32-byte aligned
  int bn;              // bf16 weights on CTA pairs: columns of a tile, 64 .. 256 in steps of 32 (see choose_pair_width)
  const uint8_t *lora_rhs;  // null = no LoRA k-block
  const float *c_scale;     // bf16 weights only: factor of the fp32 accumulator in the epilogue (null = 1)
  int expert_rows;          // grouped bf16 weights: rows of one expert's matrix in the stacked [E * rows, in] matrix
  // dX launch whose result is the gradient of the experts' hidden activation (down^T): instead of storing it, the
  // epilogue applies the SwiGLU backward to it and stores the gradients of the gate and up projections' outputs
  // (c: g_gate, sb_g_up: g_up), reading the forward's gate(x) and up(x) (sb_gate, sb_up).  bf16 only.
  const void *sb_gate;
  const void *sb_up;
  void *sb_g_up;
  int dual_k;               // bf16 weights: the reduction runs over two operand pairs, C = A.W + A2.W2 (A2 through
                            // map_h, W2 through map_l), num_kb k-blocks each
  // Fused gate/up/SwiGLU forward of a frozen expert (forward, 128-wide tiles, 16-bit outputs): a tile's
  // columns 0..63 are features [64 j, 64 j + 64) of the gate projection, columns 64..127 the same
  // features of the up projection.  c receives gate(x), c_up up(x), c_hidden silu(gate(x)) * up(x),
  // each rounded to the storage dtype the way the separate kernels round them.
  uint32_t spin_limit;   // polls of one wait before it gives up
  uint32_t stall_bytes;  // self-test only: bytes the first activation tile announces but never receives
  int swiglu;
  const uint8_t *codes_up;
  const void *scales_up;
  void *c_up;
  void *c_hidden;
};

// Grouped mode: one launch covers the same product for a run of experts whose activation rows lie
// back to back in one packed buffer (rows offsets[e] .. offsets[e+1] belong to expert e).  The table
// travels as a kernel parameter, so nothing is read back from or copied to the device to schedule it.
constexpr int MAX_GROUPS = 80;   // the table must fit the 4 KB of kernel parameters

struct GroupTable
{
  int32_t offsets[MAX_GROUPS + 1];      // first packed row of every expert
  int32_t mtile_start[MAX_GROUPS + 1];  // running count of 256-row tiles
  const uint8_t *codes[MAX_GROUPS];
  const void *scales[MAX_GROUPS];
  const uint8_t *codes_up[MAX_GROUPS];   // fused gate/up mode only
  const void *scales_up[MAX_GROUPS];
  int32_t num_groups;
};

struct NoGroupTable
{
  int32_t unused;
};

template <bool GROUPED>
struct GroupSel
{
  typedef NoGroupTable type;
};
template <>
struct GroupSel<true>
{
  typedef GroupTable type;
};

// What a tile of the schedule works on.
struct TileWork
{
  int expert;        // grouped mode: index of the expert inside this launch's table
  int n_tile;
  int64_t row0;      // first activation / output row of the tile
  int64_t row_end;   // rows at or beyond this one belong to somebody else
  const uint8_t *codes;
  const void *scales;
  const uint8_t *codes_up;
  const void *scales_up;
};

template <bool GROUPED>
__device__ __forceinline__ TileWork locate_tile(int tile, const UmmaParams &p, const typename GroupSel<GROUPED>::type &gt);

template <>
__device__ __forceinline__ TileWork locate_tile<false>(int tile, const UmmaParams &p, const NoGroupTable &)
{
  // In bands of p.band row tiles, row tiles fastest: the CTAs running at one time then work on a near-square block of
  // the output (74 pairs: 8 x 9 tiles), which takes the fewest operand bytes.  With column tiles fastest every band of
  // 256 tokens swept the whole weight, and one that does not fit L2 was read from memory again each time
  // (4096 -> 14336, 2047 tokens: 198 us, with the bands 165).
  TileWork t;
  t.expert = 0;
  const int per_band = p.band * p.num_n_tiles;
  const int band0 = tile / per_band * p.band;
  const int rows = min(p.band, p.num_m_tiles - band0);
  const int local = tile - band0 * p.num_n_tiles;
  t.n_tile = local / rows;
  t.row0 = static_cast<int64_t>(band0 + local % rows) * BM;
  t.row_end = p.m;
  t.codes = p.codes;
  t.scales = p.scales;
  t.codes_up = p.codes_up;
  t.scales_up = p.scales_up;
  return t;
}

template <>
__device__ __forceinline__ TileWork locate_tile<true>(int tile, const UmmaParams &p, const GroupTable &gt)
{
  const int mt = tile / p.num_n_tiles;   // row tile among all experts' row tiles; column tiles fastest
  int lo = 0;
  int hi = gt.num_groups;                // mtile_start[lo] <= mt < mtile_start[hi]
  while (hi - lo > 1)
  {
    const int mid = (lo + hi) >> 1;
    if (gt.mtile_start[mid] <= mt)
    {
      lo = mid;
    }
    else
    {
      hi = mid;
    }
  }
  TileWork t;
  t.expert = lo;
  t.n_tile = tile % p.num_n_tiles;
  t.row0 = static_cast<int64_t>(gt.offsets[lo]) + static_cast<int64_t>(mt - gt.mtile_start[lo]) * BM;
  t.row_end = gt.offsets[lo + 1];
  t.codes = gt.codes[lo];
  t.scales = gt.scales[lo];
  t.codes_up = gt.codes_up[lo];
  t.scales_up = gt.scales_up[lo];
  return t;
}

// 32 bytes of an output row: one store where alignment allows.  A lane owns a row, so every store instruction touches 32
// lines; with 16-byte stores their number, not the bytes, bounded the epilogue (4800 cycles a 256-wide tile).
__device__ __forceinline__ void store_row32(void *p, const uint32_t (&v)[8], bool wide)
{
  if (wide)
  {
    store_bf16x16(p, make_uint4(v[0], v[1], v[2], v[3]), make_uint4(v[4], v[5], v[6], v[7]));
  }
  else
  {
    static_cast<uint4 *>(p)[0] = make_uint4(v[0], v[1], v[2], v[3]);
    static_cast<uint4 *>(p)[1] = make_uint4(v[4], v[5], v[6], v[7]);
  }
}

__device__ __forceinline__ void load_row32(const void *p, uint32_t (&v)[8], bool wide)
{
  if (wide)
  {
    asm volatile("ld.global.nc.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "l"(p));
  }
  else
  {
    const uint4 a = __ldg(static_cast<const uint4 *>(p));
    const uint4 b = __ldg(static_cast<const uint4 *>(p) + 1);
    v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w;
    v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
  }
}

template <int WMODE, bool BWD, int BN, bool GROUPED, bool PAIR>
__global__ void __launch_bounds__(NUM_THREADS, 1)
linear_umma_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                   const __grid_constant__ CUtensorMap map_h, const __grid_constant__ CUtensorMap map_l,
                   const UmmaParams p,
                   const __grid_constant__ typename GroupSel<GROUPED>::type gt)
{
  constexpr int PLANES = planes_of(WMODE);
  constexpr bool IS_I4 = (WMODE == W_I4 || WMODE == W_I4S);
  typedef TileCfg<BN, PLANES, PAIR> Cfg;
  constexpr int MTK = Cfg::MTK;
  constexpr int BNC = Cfg::BNC;
  constexpr int A_STAGE = Cfg::A_BYTES;
  constexpr int B_PLANE_BYTES = Cfg::B_PLANE_BYTES;
  constexpr int B_STAGE_BYTES = Cfg::B_STAGE_BYTES;
  constexpr int STAGE_BYTES = Cfg::STAGE_BYTES;
  constexpr int STAGES = Cfg::STAGES;
  constexpr int ACC_COLS = Cfg::ACC_COLS;
  constexpr int ACC_BUFS = Cfg::ACC_BUFS;
  constexpr uint32_t CTAS = PAIR ? 2u : 1u;   // CTAs that work on one tile
  // columns of a tile, and weight rows of it that this CTA stages: chosen per launch where the weight is fed by copies
  // alone (the places in shared and tensor memory are those of the widest tile)
  constexpr bool ANY_WIDTH = PAIR && WMODE == W_BF16;
  const int bn = ANY_WIDTH ? p.bn : BN;
  const int bnc = ANY_WIDTH ? p.bn / 2 : BNC;
  // A bf16 weight needs no dequant warps: four of them join the epilogue, so every quarter of the accumulator's
  // lanes is drained by two warps that take alternate 32-column chunks.
  constexpr int EPI_GROUPS = (WMODE == W_BF16) ? 2 : 1;
  constexpr int DEQ_TEAMS = deq_teams(PAIR);
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t bars[MAX_STAGES * 3 + 4];
  __shared__ uint64_t drain_bar;   // give-up path only: the MMAs issued so far have completed
  __shared__ uint32_t tmem_base_slot;
  __shared__ uint32_t cta_abort;   // a wait of this CTA has run out

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  auto a_addr = [&](int s, int mt) { return smem_base + static_cast<uint32_t>(s) * STAGE_BYTES + mt * A_SUB_BYTES; };
  auto b_addr = [&](int s) { return smem_base + static_cast<uint32_t>(s) * STAGE_BYTES + A_STAGE; };
  const uint32_t bar0 = smem_u32(bars);
  auto a_full = [&](int s) { return bar0 + static_cast<uint32_t>(s) * 8u; };
  auto b_full = [&](int s) { return bar0 + static_cast<uint32_t>(STAGES + s) * 8u; };
  auto empty = [&](int s) { return bar0 + static_cast<uint32_t>(2 * STAGES + s) * 8u; };
  auto acc_full = [&](int a) { return bar0 + static_cast<uint32_t>(3 * STAGES + a) * 8u; };
  auto acc_empty = [&](int a) { return bar0 + static_cast<uint32_t>(3 * STAGES + 2 + a) * 8u; };

  // Pair mode: rank 0 of the cluster (the leader) issues the MMAs; the barriers that gate them (operands
  // landed, accumulator drained) are the leader's, and the other CTA's copies and warps arrive on them
  // through the cluster's shared address space.  The barriers that the MMAs' completion signals (stage free,
  // accumulator ready) exist in both CTAs and get a multicast commit.
  const uint32_t rank = PAIR ? cluster_ctarank() : 0u;
  const int worker = PAIR ? static_cast<int>(blockIdx.x >> 1) : static_cast<int>(blockIdx.x);
  const int workers = PAIR ? static_cast<int>(gridDim.x >> 1) : static_cast<int>(gridDim.x);
  auto lead = [&](uint32_t bar) { return PAIR ? map_to_cta(bar, 0u) : bar; };
  auto arrive_lead = [&](uint32_t bar)
  {
    if (PAIR)
    {
      mbar_arrive_cluster(map_to_cta(bar, 0u));
    }
    else
    {
      mbar_arrive(bar);
    }
  };
  volatile uint32_t *abort_word = &cta_abort;
  auto wait = [&](uint32_t bar, uint32_t parity) { return mbar_wait(bar, parity, abort_word, p.spin_limit, &g_umma_timeout_flag); };
  if (threadIdx.x == 0)
  {
    cta_abort = 0u;
    mbar_init(smem_u32(&drain_bar), 1);
    for (int s = 0; s < STAGES; ++s)
    {
      mbar_init(a_full(s), 1);
      mbar_init(b_full(s), (8 / DEQ_TEAMS) * CTAS);   // (a bf16 weight's copies arrive on a_full)
      mbar_init(empty(s), 1);
    }
    for (int a = 0; a < ACC_BUFS; ++a)
    {
      mbar_init(acc_full(a), 1);
      mbar_init(acc_empty(a), 4 * EPI_GROUPS * CTAS);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1)
  {
    if (PAIR)
    {
      // both CTAs of the pair run this, from the same warp number
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_slot)),
                   "r"(TMEM_COLS)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    else
    {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_slot)),
                   "r"(TMEM_COLS)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
  }
  tc_fence_before();
  __syncthreads();
  if (PAIR)
  {
    cluster_sync_all();   // the other CTA's barriers are initialised before anything arrives on them
  }
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_slot;
  // nothing above reads or writes what another kernel does: all of it runs beside the end of the previous one
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

  const int num_tiles = p.num_m_tiles * p.num_n_tiles;
  const int num_kb = p.k_total / BK;
  // with a LoRA product the loop runs one more k-block whose operands are the padded factors
  const int num_kb_all = (p.dual_k ? 2 * num_kb : num_kb) + ((p.lora_rhs != nullptr) ? 1 : 0);

  // One thread copies the activation tiles and, where the weight is bf16, another the weight tiles: waiting for a place,
  // announcing the bytes and issuing both copies took one thread 460 cycles a k-block, more than most tiles' MMAs take.
  // (pair: the leader announces both CTAs' bytes; the other CTA's copies may complete first, the phase cannot end before
  // the leader's arrival)
  const uint32_t lead_bar0 = lead(bar0);
  auto load = [&](uint32_t dst, const CUtensorMap *map, int c0, int c1, int stage)
  {
    if (PAIR)
    {
      tma_load_2d_pair(dst, map, c0, c1, lead_bar0 + static_cast<uint32_t>(stage) * 8u);
    }
    else
    {
      tma_load_2d(dst, map, c0, c1, a_full(stage));
    }
  };

  if (warp == 0)
  {
    // ------------------------------------------------------------ TMA producer: activations
    auto produce = [&]()
    {
      // (a bf16 weight's tile arrives on the same barrier)
      const uint32_t b_bytes = BWD ? static_cast<uint32_t>((bnc + 63) / 64) * 8192u : static_cast<uint32_t>(bnc) * 128u;
      const uint32_t bytes = (A_STAGE + (WMODE == W_BF16 ? b_bytes : 0u)) * CTAS;
      uint32_t stall = p.stall_bytes;
      int s = 0;
      uint32_t par = 0;
      for (int tile = worker; tile < num_tiles; tile += workers)
      {
        const TileWork tw = locate_tile<GROUPED>(tile, p, gt);
        const int row_tile = static_cast<int>(tw.row0) + static_cast<int>(rank) * BM_SUB;   // pair: this CTA's half
        for (int kb = 0; kb < num_kb_all; ++kb)
        {
          if (!wait(empty(s), par ^ 1u))
          {
            return;   // nothing new is started once a wait has run out
          }
          if (rank == 0)
          {
            mbar_expect_tx(a_full(s), bytes + stall);
            stall = 0;
          }
          // from num_kb on: the LoRA k-block's activation-side operand, or the second operand pair's k-blocks
          const CUtensorMap *map = (kb < num_kb) ? &map_a : &map_h;
          const int kc = (kb < num_kb) ? kb * BK : (kb - num_kb) * BK;
#pragma unroll
          for (int mt = 0; mt < MTK; ++mt)
          {
            load(a_addr(s, mt), map, kc, row_tile + mt * BM_SUB, s);
          }
          if (++s == STAGES)
          {
            s = 0;
            par ^= 1u;
          }
        }
      }
    };
    if (lane == 0)
    {
      produce();
    }
  }
  else if (WMODE == W_BF16 && warp == B_WARP)
  {
    // ------------------------------------------------------------ TMA producer: bf16 weight
    auto produce = [&]()
    {
      int s = 0;
      uint32_t par = 0;
      for (int tile = worker; tile < num_tiles; tile += workers)
      {
        const TileWork tw = locate_tile<GROUPED>(tile, p, gt);
        const int nc0 = tw.n_tile * bn + static_cast<int>(rank) * bnc;   // this CTA's weight rows
        // grouped: the experts' matrices lie stacked in one [E * rows, in] matrix
        const int erow = GROUPED ? tw.expert * p.expert_rows : 0;
        for (int kb = 0; kb < num_kb_all; ++kb)
        {
          if (!wait(empty(s), par ^ 1u))
          {
            return;
          }
          // from num_kb on: the padded LoRA factor, or the second operand pair's weight
          const CUtensorMap *map = (kb < num_kb) ? &map_b : &map_l;
          const int kc = (kb < num_kb) ? kb * BK : (kb - num_kb) * BK;
          if (!BWD && p.swiglu)
          {
            // HALF features of the gate projection (map_b) and the same features of the up projection (map_l)
            constexpr int HALF = BN / 2;
            const int f0 = erow + tw.n_tile * HALF;
            if (PAIR)
            {
              load(b_addr(s), (rank == 0) ? &map_b : &map_l, kc, f0, s);
            }
            else
            {
              load(b_addr(s), &map_b, kc, f0, s);
              load(b_addr(s) + static_cast<uint32_t>(HALF) * 128u, &map_l, kc, f0, s);
            }
          }
          else if (BWD)
          {
            // [k rows][n cols]: boxes of 64 n x 64 k land as the MN-major blocks
#pragma unroll
            for (int nb = 0; nb < BNC / 64; ++nb)
            {
              if (ANY_WIDTH && nb * 64 >= bnc)
              {
                break;
              }
              load(b_addr(s) + static_cast<uint32_t>(nb) * 8192u, map, nc0 + nb * 64, erow + kc, s);
            }
          }
          else
          {
            load(b_addr(s), map, kc, erow + nc0, s);
          }
          if (++s == STAGES)
          {
            s = 0;
            par ^= 1u;
          }
        }
      }
    };
    if (lane == 0)
    {
      produce();
    }
  }
  else if (warp == 1)
  {
    // -------------------------------------------------------------- MMA issuer
    // One elected lane does it all (of the leader CTA's warp in a pair), with as few instructions as it takes: the loop's
    // own latency, not the tensor core, bounded the kernel while the whole warp ran it with an election and a warp
    // barrier per k-block (560 cycles a k-block at any tile width; 512 is what a 256-wide tile's MMAs take).
    // After a wait that ran out it stops: a barrier that still expects bytes must not be armed again, and the producer
    // arms one only after its stage has been committed here.
    auto multiply = [&]()
    {
      const uint32_t idesc = make_idesc(BWD, bn, PAIR ? 2 * BM_SUB : BM_SUB);
      auto mma = [&](uint32_t d, uint64_t a, uint64_t b, uint32_t accumulate)
      {
        if (PAIR)
        {
          umma_bf16_pair(d, a, b, idesc, accumulate);
        }
        else
        {
          umma_bf16(d, a, b, idesc, accumulate);
        }
      };
      auto commit = [&](uint32_t bar)
      {
        if (PAIR)
        {
          umma_commit_pair(bar);
        }
        else
        {
          umma_commit(bar);
        }
      };
      const uint64_t adesc_base = make_desc(a_addr(0, 0), 16, 1024);
      const uint64_t bdesc_base = BWD ? make_desc(b_addr(0), 8192, 1024) : make_desc(b_addr(0), 16, 1024);
      int s = 0;
      uint32_t par = 0;
      int acc = 0;
      uint32_t acc_par = 0;
      for (int tile = worker; tile < num_tiles; tile += workers)
      {
        if (!wait(acc_empty(acc), acc_par ^ 1u))
        {
          return;
        }
        const uint32_t d0 = tmem_base + static_cast<uint32_t>(acc * ACC_COLS);
        uint32_t accumulate = 0;
        for (int kb = 0; kb < num_kb_all; ++kb)
        {
          if (!wait(a_full(s), par) || (WMODE != W_BF16 && !wait(b_full(s), par)))
          {
            return;
          }
          tc_fence_after();
          // descriptor address fields count 16-byte units
          const uint64_t stage = static_cast<uint64_t>(s) * (STAGE_BYTES >> 4);
#pragma unroll
          for (int mt = 0; mt < MTK; ++mt)
          {
#pragma unroll
            for (int k16 = 0; k16 < BK / UMMA_K; ++k16)
            {
              const uint64_t adesc = adesc_base + stage + static_cast<uint64_t>((mt * A_SUB_BYTES + k16 * (UMMA_K * 2)) >> 4);
              const uint64_t bdesc = bdesc_base + stage + static_cast<uint64_t>((BWD ? k16 * 2048 : k16 * (UMMA_K * 2)) >> 4);
              mma(d0 + static_cast<uint32_t>(mt * BN), adesc, bdesc, (k16 == 0) ? accumulate : 1u);
              if (PLANES == 2 && kb < num_kb)
              {
                // the low-order term of the weights (the LoRA k-block has one plane only)
                mma(d0 + static_cast<uint32_t>(mt * BN), adesc, bdesc + static_cast<uint64_t>(B_PLANE_BYTES >> 4), 1u);
              }
            }
          }
          commit(empty(s));
          accumulate = 1;
          if (++s == STAGES)
          {
            s = 0;
            par ^= 1u;
          }
        }
        commit(acc_full(acc));
        if (++acc == ACC_BUFS)
        {
          acc = 0;
          acc_par ^= 1u;
        }
      }
    };
    if (rank == 0 && elect_one())
    {
      multiply();
    }
    __syncwarp();
  }
  else if (warp >= 2 && warp < DEQ_WARP0 + 4 * (EPI_GROUPS - 1))
  {
    // ---------------------------------------------------------------- epilogue
    const int quarter = warp & 3;  // TMEM lanes 32*quarter .. +31 are the ones this warp may read
    const int epi_group = (warp - 2) >> 2;   // 0, or 1 for the warps that joined from the dequant role
    int acc = 0;
    uint32_t acc_par = 0;
    for (int tile = worker; tile < num_tiles; tile += workers)
    {
      const TileWork tw = locate_tile<GROUPED>(tile, p, gt);
      const int n_tile = tw.n_tile;
      float out_scale = 1.0f;
      if ((WMODE == W_I8 || (WMODE == W_BF16 && GROUPED)) && tw.scales != nullptr)
      {
        // (grouped bf16 weights: expanded int8 codes, whose per-tensor scale the table still carries)
        out_scale = __ldg(static_cast<const float *>(tw.scales));
      }
      if (WMODE == W_BF16 && p.c_scale != nullptr)
      {
        out_scale = __ldg(p.c_scale);
      }
      wait(acc_full(acc), acc_par);
      tc_fence_after();
      if (!BWD && (BN == 128 || PAIR) && p.swiglu)
      {
        constexpr int HALF = BN / 2;   // features of each projection in a tile
        float up_scale = 1.0f;
        if ((WMODE == W_I8 || (WMODE == W_BF16 && GROUPED)) && tw.scales_up != nullptr)
        {
          up_scale = __ldg(static_cast<const float *>(tw.scales_up));
        }
        const int hid = p.n_total / 2;   // features per projection
#pragma unroll
        for (int mt = 0; mt < MTK; ++mt)
        {
          const int64_t row = tw.row0 + static_cast<int64_t>(rank) * BM_SUB + mt * BM_SUB + quarter * 32 + lane;
#pragma unroll
          for (int cb = 0; cb < HALF / 32; ++cb)
          {
            if (EPI_GROUPS > 1 && (cb % EPI_GROUPS) != epi_group)
            {
              continue;
            }
            uint32_t rg[32];
            uint32_t ru[32];
            const uint32_t tbase = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) +
                                   static_cast<uint32_t>(acc * ACC_COLS + mt * BN);
            tmem_ld32(tbase + cb * 32, rg);
            tmem_ld32(tbase + HALF + cb * 32, ru);
            tmem_ld_wait();
            if (row < tw.row_end)
            {
              const int64_t off = row * hid + static_cast<int64_t>(n_tile) * HALF + cb * 32;
              uint4 *dg = reinterpret_cast<uint4 *>(static_cast<uint16_t *>(p.c) + off);
              uint4 *du = reinterpret_cast<uint4 *>(static_cast<uint16_t *>(p.c_up) + off);
              uint4 *dh = reinterpret_cast<uint4 *>(static_cast<uint16_t *>(p.c_hidden) + off);
#pragma unroll
              for (int q = 0; q < 2; ++q)
              {
                uint32_t pg[8], pu[8], ph[8];
#pragma unroll
                for (int e = 0; e < 8; ++e)
                {
                  float g2[2], u2[2], h2[2];
#pragma unroll
                  for (int z = 0; z < 2; ++z)
                  {
                    // the separate kernels' roundings: projection outputs to the storage dtype,
                    // silu(gate) to the storage dtype, then the product
                    g2[z] = round_through<CAIFQ_BF16>(__uint_as_float(rg[16 * q + 2 * e + z]) * out_scale);
                    u2[z] = round_through<CAIFQ_BF16>(__uint_as_float(ru[16 * q + 2 * e + z]) * up_scale);
                    const float act = round_through<CAIFQ_BF16>(g2[z] / (1.0f + expf(-g2[z])));
                    h2[z] = act * u2[z];
                  }
                  pg[e] = pack_bf16x2(g2[0], g2[1]);
                  pu[e] = pack_bf16x2(u2[0], u2[1]);
                  ph[e] = pack_bf16x2(h2[0], h2[1]);
                }
                store_row32(dg + 2 * q, pg, p.wide_stores != 0);
                store_row32(du + 2 * q, pu, p.wide_stores != 0);
                store_row32(dh + 2 * q, ph, p.wide_stores != 0);
              }
            }
          }
        }
      }
      else if (BWD && p.sb_gate != nullptr)
      {
        // g_hidden = round(acc); g_up = round(g_hidden * round(silu(gate))); g_gate = round(round(g_hidden *
        // up) * silu'(gate)): the separate kernel's rounding points (see swiglu_bwd_kernel).  Sixteen columns at a time:
        // 32-byte loads and stores, and no more registers than that takes.
#pragma unroll
        for (int mt = 0; mt < MTK; ++mt)
        {
          const int64_t row = tw.row0 + static_cast<int64_t>(rank) * BM_SUB + mt * BM_SUB + quarter * 32 + lane;
          for (int cb = epi_group; cb < bn / 16; cb += EPI_GROUPS)
          {
            const int64_t off = row * p.n_total + static_cast<int64_t>(n_tile) * bn + cb * 16;
            const bool mine = row < tw.row_end && n_tile * bn + cb * 16 < p.n_total;
            uint32_t gw[8] = {}, uw[8] = {};
            if (mine)
            {
              load_row32(static_cast<const uint16_t *>(p.sb_gate) + off, gw, p.wide_stores != 0);
              load_row32(static_cast<const uint16_t *>(p.sb_up) + off, uw, p.wide_stores != 0);
            }
            uint32_t r[16];
            tmem_ld16(tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) +
                          static_cast<uint32_t>(acc * ACC_COLS + mt * BN + cb * 16),
                      r);
            tmem_ld_wait();
            if (mine)
            {
#pragma unroll
              for (int e = 0; e < 8; ++e)
              {
                float og[2], ou[2];
#pragma unroll
                for (int z = 0; z < 2; ++z)
                {
                  const float x = z ? __uint_as_float(gw[e] & 0xFFFF0000u) : __uint_as_float(gw[e] << 16);
                  const float uv = z ? __uint_as_float(uw[e] & 0xFFFF0000u) : __uint_as_float(uw[e] << 16);
                  const float gh = round_through<CAIFQ_BF16>(__uint_as_float(r[2 * e + z]) * out_scale);
                  // one fast exponential and one fast reciprocal per element: 256 x 128 elements per tile must
                  // fit beside the next tile's MMAs (the exact expf and two IEEE divisions did not: 2x slower);
                  // fp32 relative error ~1e-6 before the bf16 roundings
                  const float sg = __fdividef(1.0f, 1.0f + __expf(-x));
                  const float act = round_through<CAIFQ_BF16>(x * sg);
                  ou[z] = gh * act;
                  const float gv = round_through<CAIFQ_BF16>(gh * uv);
                  og[z] = gv * sg * fmaf(x, 1.0f - sg, 1.0f);
                }
                gw[e] = pack_bf16x2(og[0], og[1]);
                uw[e] = pack_bf16x2(ou[0], ou[1]);
              }
              store_row32(static_cast<uint16_t *>(p.c) + off, gw, p.wide_stores != 0);
              store_row32(static_cast<uint16_t *>(p.sb_g_up) + off, uw, p.wide_stores != 0);
            }
          }
        }
      }
      else
#pragma unroll
      for (int mt = 0; mt < MTK; ++mt)
      {
        const int64_t row = tw.row0 + static_cast<int64_t>(rank) * BM_SUB + mt * BM_SUB + quarter * 32 + lane;
#pragma unroll
        for (int cb = 0; cb < BN / 32; ++cb)
        {
          if ((EPI_GROUPS > 1 && (cb % EPI_GROUPS) != epi_group) || (ANY_WIDTH && cb * 32 >= bn))
          {
            continue;
          }
          uint32_t r[32];
          const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) +
                                 static_cast<uint32_t>(acc * ACC_COLS + mt * BN + cb * 32);
          tmem_ld32(taddr, r);
          tmem_ld_wait();
          // (the last column tile may reach past the output's width when the width is not a multiple of the
          // tile's: those columns, computed on zero or foreign weight rows, are not stored)
          if (row < tw.row_end && n_tile * bn + cb * 32 < p.n_total)
          {
            const int64_t off = row * p.n_total + static_cast<int64_t>(n_tile) * bn + cb * 32;
            if (p.c_dtype == CAIFQ_F32)
            {
              float4 *dst = reinterpret_cast<float4 *>(static_cast<float *>(p.c) + off);
#pragma unroll
              for (int q = 0; q < 4; ++q)
              {
                uint32_t v[8];
#pragma unroll
                for (int e = 0; e < 8; ++e)
                {
                  v[e] = __float_as_uint(__uint_as_float(r[8 * q + e]) * out_scale);
                }
                if (p.accumulate)
                {
                  const float4 o0 = dst[2 * q];
                  const float4 o1 = dst[2 * q + 1];
                  const float o[8] = {o0.x, o0.y, o0.z, o0.w, o1.x, o1.y, o1.z, o1.w};
#pragma unroll
                  for (int e = 0; e < 8; ++e)
                  {
                    v[e] = __float_as_uint(__uint_as_float(v[e]) + o[e]);
                  }
                }
                store_row32(dst + 2 * q, v, p.wide_stores != 0);
              }
            }
            else
            {
              // 16-bit outputs: 32 values = 64 bytes = two 32-byte stores
              uint4 *dst = reinterpret_cast<uint4 *>(static_cast<uint16_t *>(p.c) + off);
#pragma unroll
              for (int q = 0; q < 2; ++q)
              {
                float v[16];
#pragma unroll
                for (int e = 0; e < 16; ++e)
                {
                  v[e] = __uint_as_float(r[16 * q + e]) * out_scale;
                }
                uint32_t packed[8];
                if (p.accumulate)
                {
                  const uint4 o0 = dst[2 * q];
                  const uint4 o1 = dst[2 * q + 1];
                  const uint32_t ow[8] = {o0.x, o0.y, o0.z, o0.w, o1.x, o1.y, o1.z, o1.w};
#pragma unroll
                  for (int e = 0; e < 8; ++e)
                  {
                    float lo;
                    float hi;
                    if (p.c_dtype == CAIFQ_BF16)
                    {
                      lo = __uint_as_float(ow[e] << 16);
                      hi = __uint_as_float(ow[e] & 0xFFFF0000u);
                      v[2 * e] = round_through<CAIFQ_BF16>(v[2 * e]) + lo;
                      v[2 * e + 1] = round_through<CAIFQ_BF16>(v[2 * e + 1]) + hi;
                    }
                    else
                    {
                      const __half2 h = *reinterpret_cast<const __half2 *>(&ow[e]);
                      v[2 * e] = round_through<CAIFQ_F16>(v[2 * e]) + __low2float(h);
                      v[2 * e + 1] = round_through<CAIFQ_F16>(v[2 * e + 1]) + __high2float(h);
                    }
                  }
                }
#pragma unroll
                for (int e = 0; e < 8; ++e)
                {
                  if (p.c_dtype == CAIFQ_BF16)
                  {
                    packed[e] = pack_bf16x2(v[2 * e], v[2 * e + 1]);
                  }
                  else
                  {
                    const __half2 h = __floats2half2_rn(v[2 * e], v[2 * e + 1]);
                    packed[e] = *reinterpret_cast<const uint32_t *>(&h);
                  }
                }
                store_row32(dst + 2 * q, packed, p.wide_stores != 0);
              }
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0)
      {
        arrive_lead(acc_empty(acc));
      }
      if (++acc == ACC_BUFS)
      {
        acc = 0;
        acc_par ^= 1u;
      }
    }
  }
  else if (WMODE != W_BF16)
  {
    // ------------------------------------------------------ weight dequantization
    // The eight warps work as DEQ_TEAMS teams; team t converts the k-blocks whose number is t modulo
    // DEQ_TEAMS, so with two teams a k-block's conversion (loads, ~150 instructions per thread, stores,
    // proxy fence, barrier arrive) has two k-blocks of MMA time to finish in.
    constexpr int TEAM_THREADS = DEQ_THREADS / DEQ_TEAMS;
    const int team = (threadIdx.x - DEQ_WARP0 * 32) / TEAM_THREADS;
    const int d = (threadIdx.x - DEQ_WARP0 * 32) % TEAM_THREADS;
    // 16-byte chunks of codes per k-block and thread, and where they go:
    //   forward  (K-major B): tile rows are n, a chunk is 16 B of one row's k range
    //   backward (MN-major B): tile rows are k, a chunk is 16 B of one k-row's n range
    constexpr int ELEMS = (WMODE == W_I8) ? 16 : 32;                 // codes per chunk
    constexpr int CHUNKS = (BNC * BK) / ELEMS;                       // per k-block (of this CTA's weight rows)
    constexpr int PER_THREAD = CHUNKS / TEAM_THREADS;
    constexpr int CHUNKS_PER_ROW = (BWD ? BNC : BK) / ELEMS;         // chunks along the contiguous direction
    static_assert(PER_THREAD >= 1, "tile too small for the dequant warps");

    uint32_t gkb0 = 0;   // k-blocks (of all tiles so far) before this tile: the ring position of its first one
    for (int tile = worker; tile < num_tiles; tile += workers, gkb0 += static_cast<uint32_t>(num_kb_all))
    {
      const TileWork tw = locate_tile<GROUPED>(tile, p, gt);
      const int n_tile = tw.n_tile;
      const int n0 = n_tile * BN + static_cast<int>(rank) * BNC;   // first of this CTA's weight rows / columns
      // chunk -> (row inside the tile, part along the contiguous direction)
      int c_row[PER_THREAD];
      int c_part[PER_THREAD];
#pragma unroll
      for (int i = 0; i < PER_THREAD; ++i)
      {
        const int c = d + i * TEAM_THREADS;
        if (BWD)
        {
          // A chunk expands to 64 (int4) or 32 (int8) bytes of one 128-byte operand row, whose 16-byte
          // pieces sit at (piece ^ row % 8).  Eight consecutive threads (one shared-memory store phase)
          // take RPQ neighbouring rows x PPQ neighbouring chunks: eight distinct bank groups, and the
          // PPQ chunks of a row are contiguous in global memory.
          constexpr int PPQ = 128 / (ELEMS * 2);
          constexpr int RPQ = 8 / PPQ;
          const int lo = c & 7;
          const int hi = c >> 3;
          c_row[i] = (hi % (BK / RPQ)) * RPQ + lo / PPQ;
          c_part[i] = (hi / (BK / RPQ)) * PPQ + lo % PPQ;
        }
        else
        {
          c_row[i] = c / CHUNKS_PER_ROW;
          c_part[i] = c % CHUNKS_PER_ROW;
        }
      }
      auto load = [&](int kb, uint4 (&raw)[PER_THREAD], float (&sc)[PER_THREAD])
      {
        const int k0 = kb * BK;
#pragma unroll
        for (int i = 0; i < PER_THREAD; ++i)
        {
          // element coordinates of the chunk's first code in the [out, in] matrix
          int64_t o = BWD ? (k0 + c_row[i]) : (n0 + c_row[i]);
          const uint8_t *codes = tw.codes;
          const void *scales = tw.scales;
          if (!BWD && p.swiglu)
          {
            // first half of the tile's rows: gate features HALF j + r; second half: the same up features
            constexpr int HALF = BN / 2;
            const int t = static_cast<int>(rank) * BNC + c_row[i];
            o = static_cast<int64_t>(n_tile) * HALF + (t % HALF);
            if (t >= HALF)
            {
              codes = tw.codes_up;
              scales = tw.scales_up;
            }
          }
          const int64_t ii = BWD ? (n0 + c_part[i] * ELEMS) : (k0 + c_part[i] * ELEMS);
          const int64_t flat = o * p.in_dim + ii;
          const uint8_t *src = codes + ((WMODE == W_I8) ? flat : (flat >> 1));
          raw[i] = __ldg(reinterpret_cast<const uint4 *>(src));
          if (IS_I4)
          {
            // in_dim is a multiple of the group size here, so the flat group index splits into a row
            // part and a 32-bit division inside the row (a 64-bit division costs as much as the conversion)
            const int64_t grp = o * p.groups_per_row + static_cast<int>(ii) / p.group_size;
            sc[i] = __half2float(static_cast<const __half *>(scales)[grp]);
          }
          else
          {
            sc[i] = 1.0f;
          }
        }
      };

      // this team's first k-block of the tile
      const int kb_first = static_cast<int>((static_cast<uint32_t>(team) + DEQ_TEAMS - (gkb0 % DEQ_TEAMS)) % DEQ_TEAMS);
      // With eight chunks per thread the next block's codes are not kept in flight beside the current
      // ones (registers); the other team's block covers the load instead.
      constexpr bool PREFETCH = PER_THREAD <= 4;
      uint4 raw[PER_THREAD];
      float sc[PER_THREAD];
      if (PREFETCH && kb_first < num_kb)
      {
        load(kb_first, raw, sc);
      }
      for (int kb = kb_first; kb < num_kb; kb += DEQ_TEAMS)
      {
        uint4 nraw[PER_THREAD];
        float nsc[PER_THREAD];
        if (!PREFETCH)
        {
          load(kb, raw, sc);
        }
        else if (kb + DEQ_TEAMS < num_kb)
        {
          load(kb + DEQ_TEAMS, nraw, nsc);  // in flight while this block is converted
        }
        const uint32_t gkb = gkb0 + static_cast<uint32_t>(kb);
        const int s = static_cast<int>(gkb % STAGES);
        const uint32_t par = (gkb / STAGES) & 1u;
        wait(empty(s), par ^ 1u);
        const uint32_t bbase = b_addr(s);
#pragma unroll
        for (int i = 0; i < PER_THREAD; ++i)
        {
          const uint32_t words[4] = {raw[i].x, raw[i].y, raw[i].z, raw[i].w};
          // bf16 output: ELEMS values = ELEMS/8 chunks of 16 bytes
          uint32_t outw[ELEMS / 2];
          uint32_t outl[(WMODE == W_I4S) ? ELEMS / 2 : 1];   // low-order plane (split mode)
          if (WMODE == W_I8)
          {
#pragma unroll
            for (int w = 0; w < 4; ++w)
            {
              int8x4_to_bf16(words[w], outw[2 * w], outw[2 * w + 1]);
            }
          }
          else if (WMODE == W_I4S)
          {
#pragma unroll
            for (int w = 0; w < 4; ++w)
            {
              uint32_t h4[4];
              uint32_t l4[4];
              int4x8_to_bf16_split(words[w], sc[i], h4, l4);
#pragma unroll
              for (int q = 0; q < 4; ++q)
              {
                outw[4 * w + q] = h4[q];
                outl[(WMODE == W_I4S) ? (4 * w + q) : 0] = l4[q];
              }
            }
          }
          else
          {
#pragma unroll
            for (int w = 0; w < 4; ++w)
            {
              uint32_t o4[4];
              int4x8_to_bf16(words[w], pack_bf16x2(sc[i], sc[i]), o4);
              outw[4 * w + 0] = o4[0];
              outw[4 * w + 1] = o4[1];
              outw[4 * w + 2] = o4[2];
              outw[4 * w + 3] = o4[3];
            }
          }
          const int r = c_row[i];
          const int first = c_part[i] * (ELEMS / 8);  // first 16-byte bf16 chunk along the contiguous direction
#pragma unroll
          for (int j = 0; j < ELEMS / 8; ++j)
          {
            const int cb = first + j;
            uint32_t dst;
            if (BWD)
            {
              // MN-major: 64-wide n blocks (8 KB apart), 8-row k groups (1 KB), 128-byte rows, 16-byte chunks XOR row%8
              dst = bbase + static_cast<uint32_t>((cb >> 3) * 8192 + (r >> 3) * 1024 + (r & 7) * 128 +
                                                  (((cb & 7) ^ (r & 7)) << 4));
            }
            else
            {
              // K-major: rows n of 128 bytes, 16-byte chunks XOR row%8
              dst = bbase + static_cast<uint32_t>(r * 128 + ((cb ^ (r & 7)) << 4));
            }
            asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(dst), "r"(outw[4 * j + 0]),
                         "r"(outw[4 * j + 1]), "r"(outw[4 * j + 2]), "r"(outw[4 * j + 3])
                         : "memory");
            if (WMODE == W_I4S)
            {
              constexpr int L = (WMODE == W_I4S) ? 1 : 0;
              asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(dst + static_cast<uint32_t>(B_PLANE_BYTES)),
                           "r"(outl[L * (4 * j + 0)]), "r"(outl[L * (4 * j + 1)]), "r"(outl[L * (4 * j + 2)]),
                           "r"(outl[L * (4 * j + 3)])
                           : "memory");
            }
          }
        }
        fence_proxy_async();
        __syncwarp();
        if (lane == 0)
        {
          arrive_lead(b_full(s));
        }
        if (PREFETCH)
        {
#pragma unroll
          for (int i = 0; i < PER_THREAD; ++i)
          {
            raw[i] = nraw[i];
            sc[i] = nsc[i];
          }
        }
      }
      if (p.lora_rhs != nullptr && ((gkb0 + static_cast<uint32_t>(num_kb)) % DEQ_TEAMS) == static_cast<uint32_t>(team))
      {
        // LoRA k-block (number num_kb, so one team's): the padded factor is bf16 already; copy its
        // tile into the operand layout
        const uint32_t gkb = gkb0 + static_cast<uint32_t>(num_kb);
        const int s = static_cast<int>(gkb % STAGES);
        const uint32_t par = (gkb / STAGES) & 1u;
        wait(empty(s), par ^ 1u);
        const uint32_t bbase = b_addr(s);
#pragma unroll
        for (int i = 0; i < (BNC * BK * 2 / 16) / TEAM_THREADS; ++i)
        {
          const int c = d + i * TEAM_THREADS;  // 16-byte chunk of the BNC x 64 bf16 tile
          uint32_t dst;
          const uint8_t *src;
          if (BWD)
          {
            const int r = c / (BNC / 8);   // k row (0..63) of the [64, N] factor
            const int cb = c % (BNC / 8);  // 16-byte chunk along n
            src = p.lora_rhs + (static_cast<int64_t>(r) * p.n_total + n0 + cb * 8) * 2;
            dst = bbase + static_cast<uint32_t>((cb >> 3) * 8192 + (r >> 3) * 1024 + (r & 7) * 128 +
                                                (((cb & 7) ^ (r & 7)) << 4));
          }
          else
          {
            const int r = c >> 3;  // n row (0..127) of the [N, 64] factor
            const int cb = c & 7;
            src = p.lora_rhs + (static_cast<int64_t>(n0 + r) * 64 + cb * 8) * 2;
            dst = bbase + static_cast<uint32_t>(r * 128 + ((cb ^ (r & 7)) << 4));
          }
          const uint4 v = __ldg(reinterpret_cast<const uint4 *>(src));
          asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(dst), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w)
                       : "memory");
        }
        fence_proxy_async();
        __syncwarp();
        if (lane == 0)
        {
          arrive_lead(b_full(s));
        }
      }
    }
  }

  // ------------------------------------------------------------------ teardown
  uint32_t gave_up = *abort_word;
  if (PAIR)
  {
    // every role of both CTAs has left its loops; a give-up in either CTA is handled by both
    cluster_sync_all();
    gave_up |= ld_shared_cluster(map_to_cta(smem_u32(&cta_abort), rank ^ 1u));
  }
  if (gave_up != 0u && warp == 0 && lane == 0)
  {
    // activation tiles that were started may still be on their way: give them time to land before the
    // CTA's shared memory goes back (a copy must not arrive in memory that belongs to another CTA)
    for (int i = 0; i < 64; ++i)
    {
      __nanosleep(2000);
    }
  }
  if (gave_up != 0u && warp == 1 && rank == 0)
  {
    // MMAs issued after the give-up may still run: tensor memory is released only after they have
    // completed (a commit tracks every MMA issued before it); bounded like every other wait
    if (elect_one())
    {
      if (PAIR)
      {
        umma_commit_pair_local(smem_u32(&drain_bar));
      }
      else
      {
        umma_commit(smem_u32(&drain_bar));
      }
    }
    __syncwarp();
    const uint32_t addr = smem_u32(&drain_bar);
    bool done = false;
    for (uint32_t spin = 0; spin < p.spin_limit && !done; ++spin)
    {
      uint32_t ok;
      asm volatile(
          "{\n\t.reg .pred p;\n\t"
          "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
          "selp.u32 %0, 1, 0, p;\n\t}"
          : "=r"(ok)
          : "r"(addr), "r"(0u)
          : "memory");
      done = ok != 0;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (PAIR)
  {
    // neither CTA's shared or tensor memory is touched by the other one after this
    cluster_sync_all();
  }
  if (warp == 1)
  {
    tc_fence_after();
    if (PAIR)
    {
      asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
    }
    else
    {
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
    }
  }
}

// ------------------------------------------------------------------ host side
// A host that runs a collective beside these persistent kernels leaves it some SMs: a CTA here takes
// a whole SM, and one that finds its SM taken waits for the collective to end.
int sm_count_umma() { return persistent_ctas("CAIFQ_UMMA_CTAS"); }

// CTA pairs that a launch may use (a pair takes the two SMs of one TPC)
int pair_count_umma() { return sm_count_umma() / 2; }

// smallest number of resident pairs any pair-mode kernel reported for a device so far (0 = none launched yet)
std::atomic<int> g_pair_capacity[kMaxDevices];

// Whether 256-wide tiles go to CTA pairs or to single CTAs.  Measured on 4096 x 4096, 8192 tokens, TFLOP/s: a bf16
// weight (operand fed by copies alone) 1433-1546 on pairs, 1262-1383 on single CTAs; a
// quantized weight is no faster on pairs (int8 992-1152 against 1133-1296, int4 974-1068 against
// 1069-1210): there the dequant warps' work per flop is the same in both forms and it, not the operand traffic,
// is the limit.  So pairs are the default for bf16 weights only; CAIFQ_UMMA_PAIR=1 / 0 forces them on / off.
bool pairs_enabled(int mode)
{
  if (pair_count_umma() < 1)
  {
    return false;   // a limit of one CTA leaves no pair
  }
  const char *e = std::getenv("CAIFQ_UMMA_PAIR");
  if (e == nullptr)
  {
    return mode == W_BF16;
  }
  return std::atoi(e) != 0;
}

template <int WMODE, bool BWD, int BN, bool GROUPED, bool PAIR = false>
int launch_inst(const CUtensorMap &map_a, const CUtensorMap &map_b, const CUtensorMap &map_h, const CUtensorMap &map_l,
                const UmmaParams &p,
                const typename GroupSel<GROUPED>::type &gt, cudaStream_t s)
{
  auto kernel = linear_umma_kernel<WMODE, BWD, BN, GROUPED, PAIR>;
  constexpr int SMEM_BYTES = TileCfg<BN, planes_of(WMODE), PAIR>::SMEM_BYTES;
  static std::atomic<bool> configured[kMaxDevices];
  int dev = 0;
  CAIFQ_CHECK_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices)
  {
    set_error("frozen linear (umma): device ordinal %d out of range", dev);
    return CAIFQ_ERR_UNSUPPORTED;
  }
  if (!configured[dev].load(std::memory_order_acquire))
  {
    CAIFQ_CHECK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
    configured[dev].store(true, std::memory_order_release);
  }
  const int64_t tiles = static_cast<int64_t>(p.num_m_tiles) * p.num_n_tiles;
  if (PAIR)
  {
    cudaLaunchConfig_t cfg{};
    cfg.blockDim = dim3(NUM_THREADS, 1, 1);
    cfg.dynamicSmemBytes = SMEM_BYTES;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    // The grid is persistent, so it must not hold more pairs than the device keeps resident at a time (a
    // pair that waited for another one to finish would double the launch's time): ask once per device.
    static std::atomic<int> resident[kMaxDevices];
    int cap = resident[dev].load(std::memory_order_acquire);
    if (cap == 0)
    {
      cfg.gridDim = dim3(static_cast<unsigned>(2 * (device_sm_count() / 2)), 1, 1);
      int clusters = 0;
      CAIFQ_CHECK_CUDA(cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg));
      cap = clusters > 0 ? clusters : 1;
      resident[dev].store(cap, std::memory_order_release);
      int seen = g_pair_capacity[dev].load(std::memory_order_relaxed);
      while ((seen == 0 || cap < seen) && !g_pair_capacity[dev].compare_exchange_weak(seen, cap))
      {
      }
    }
    int pairs = pair_count_umma() < cap ? pair_count_umma() : cap;
    if (tiles < pairs)
    {
      pairs = static_cast<int>(tiles);
    }
    cfg.gridDim = dim3(static_cast<unsigned>(2 * pairs), 1, 1);
    cfg.numAttrs = dependent_launches() ? 2 : 1;
    CAIFQ_CHECK_CUDA(cudaLaunchKernelEx(&cfg, kernel, map_a, map_b, map_h, map_l, p, gt));
    return CAIFQ_OK;
  }
  const int grid = tiles < sm_count_umma() ? static_cast<int>(tiles) : sm_count_umma();
  CAIFQ_CHECK_CUDA(launch_dependent(kernel, dim3(grid), dim3(NUM_THREADS), SMEM_BYTES, s, map_a, map_b, map_h, map_l, p, gt));
  return CAIFQ_OK;
}

}  // namespace

int umma_pair_capacity()
{
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices)
  {
    cudaGetLastError();
    return 0;
  }
  return g_pair_capacity[dev].load(std::memory_order_relaxed);
}

namespace
{

// Columns of a pair's tile for a bf16 weight.  The grid is persistent, so a launch takes as many waves as the busiest pair
// has tiles, and a last wave of a few tiles costs as much as a full one: 8 x 56 tiles of 256 are 6.05 waves of 74 pairs,
// 8 x 64 tiles of 224 are 6.92 (2047 tokens of 4096 -> 14336: 165 and 153 us).  A wave's time is near linear in the width
// with a constant that is the copies' (measured per wave: 15.6 us at 128 columns, 17.0 at 160, 18.4 at 192, 21.9 at 224,
// 23.5 at 256; k = 4096, so at other k the constant is the same share of a wave's copies, not of its start); few tiles (1
// wave at any width) so take the narrowest.  The grouped launches keep 256.
constexpr int kWaveConstant = 120;   // columns

int64_t pair_cost(int m_tiles, int n_total, int pairs, int bn)
{
  const int64_t tiles = static_cast<int64_t>(m_tiles) * ((n_total + bn - 1) / bn);
  return (tiles + pairs - 1) / pairs * (bn + kWaveConstant);
}

int choose_pair_width(int m_tiles, int n_total, int pairs)
{
  const int widest = n_total < 256 ? (n_total + 31) & ~31 : 256;
  int best = 0;
  int64_t best_cost = 0;
  for (int bn = widest; bn >= 64; bn -= 32)
  {
    const int64_t cost = pair_cost(m_tiles, n_total, pairs, bn);
    if (best == 0 || cost < best_cost)
    {
      best = bn;
      best_cost = cost;
    }
    if (bn <= 128)
    {
      break;   // below, the copies are all there is to a wave
    }
  }
  return best == 0 ? 64 : best;
}

}  // namespace

bool umma_supported(const LinearArgs &g)
{
  const caifq_weight &w = g.w;
  // (calls of up to 16 tokens are the few-token kernel's; from 17 on one 256-row tile, mostly
  // zero rows, still beats the fp32-FMA kernel by far)
  if (g.a_dtype != CAIFQ_BF16 || g.a_prescale != 1.0f || g.m < 17)
  {
    return false;
  }
  const int n_total = g.backward ? w.in_dim : w.out_dim;
  const int k_total = g.backward ? w.out_dim : w.in_dim;
  // (narrower or ragged outputs of a bf16 weight -- routers -- are linear_rows_kernel's: the accumulation over all of k in
  // the tensor core is five times further from 64 bits than an fp32 GEMM there, 2.1e-6 against 3.9e-7 at k = 2048)
  if ((n_total % 128) != 0 || (k_total % BK) != 0)
  {
    return false;
  }
  if ((reinterpret_cast<uintptr_t>(g.a) & 15u) != 0 || (reinterpret_cast<uintptr_t>(g.c) & 15u) != 0 ||
      (reinterpret_cast<uintptr_t>(w.codes) & 15u) != 0)
  {
    return false;
  }
  switch (w.storage)
  {
    case CAIFQ_I8:
      // per-tensor scale (or none) factors out of the product: exact for fp32 and bf16 compute
      if (w.scales != nullptr && w.scheme != CAIFQ_PER_TENSOR)
      {
        return false;
      }
      return g.compute_dtype == CAIFQ_BF16 || g.compute_dtype == CAIFQ_F32;
    case CAIFQ_I4:
      // bf16 compute: code * bf16(scale), 2^-9 from the reference's bf16(scale * code); fp32 compute: scale*code
      // as two bf16 terms (2^-17 relative), within the fp32 tolerance
      if ((g.compute_dtype != CAIFQ_BF16 && g.compute_dtype != CAIFQ_F32) || w.scales == nullptr)
      {
        return false;
      }
      return (w.group_size % 32) == 0 && (w.in_dim % w.group_size) == 0;
    case CAIFQ_BF16:
      // bf16 x bf16 products are exact in fp32
      return g.compute_dtype == CAIFQ_BF16 || g.compute_dtype == CAIFQ_F32;
    default:
      return false;
  }
}

// Whether a product of an int8 / int4 weight that may expand it first gains by that.  Both forms take time in proportion to
// k, so k does not enter.  Converting in the kernel takes 9.2 ns a k and wave of 128-wide tiles (int8 8.0 to 9.5); the
// expansion 0.43 ps a weight (int8 0.56) and the product on it 4.1 ns a k and wave of 128-wide tiles on pairs.  So it does
// not pay where the tiles are one wave of the SMs and two of the pairs.  us, converting / expanded, int4 and int8:
//   14336 columns, k 4096: 128 rows 39 / 61 and 34 / 60, 256 rows 41 / 60 and 35 / 60, 512 rows 74 / 74 and 65 / 74
//   4096 columns, k 4096: 128 rows 37 / 27 and 32 / 26, 512 rows 38 / 27 and 34 / 27
//   4096 columns, k 14336: 128 rows 117 / 85 and 95 / 84; with an adapter, 1024 rows, k 4096: 51 / 45 and 49 / 43
// Where the converting form takes 256-wide tiles (more tokens) it never won by more than a few percent.
bool umma_expansion_pays(const LinearArgs &g)
{
  const int pairs = pair_count_umma();
  const int n_total = g.backward ? g.w.in_dim : g.w.out_dim;
  const int m_tiles = static_cast<int>((g.m + BM - 1) / BM);
  if (!pairs_enabled(W_BF16) ||
      ((n_total % 256) == 0 && static_cast<int64_t>(m_tiles) * (n_total / 256) >= sm_count_umma()))
  {
    return true;
  }
  const bool i8 = g.w.storage == CAIFQ_I8;
  const int64_t tiles = static_cast<int64_t>(m_tiles) * ((n_total + 127) / 128);
  const double converting = 9.2 * static_cast<double>((tiles + sm_count_umma() - 1) / sm_count_umma());
  const int bn = choose_pair_width(m_tiles, n_total, pairs);
  const double product = 4.1 * static_cast<double>(pair_cost(m_tiles, n_total, pairs, bn)) / (128 + kWaveConstant);
  return (i8 ? 0.56e-3 : 0.43e-3) * n_total + product < converting;
}

int launch_linear_umma(const LinearArgs &g, cudaStream_t s)
{
  const caifq_weight &w = g.w;
  UmmaParams p{};
  p.spin_limit = kSpinLimit;
  p.stall_bytes = 0;
  if (take_umma_stall())
  {
    // self-test of the give-up path: the first activation tile announces 16 bytes that never arrive
    p.spin_limit = kSpinLimitTest;
    p.stall_bytes = 16;
  }
  p.codes = static_cast<const uint8_t *>(w.codes);
  p.scales = w.scales;
  p.c = g.c;
  p.c_dtype = g.c_dtype;
  p.accumulate = g.accumulate ? 1 : 0;
  p.m = g.m;
  p.n_total = g.backward ? w.in_dim : w.out_dim;
  p.k_total = g.backward ? w.out_dim : w.in_dim;
  p.in_dim = w.in_dim;
  p.group_size = w.group_size;
  p.groups_per_row = (w.group_size > 0) ? w.in_dim / w.group_size : 0;
  p.num_m_tiles = static_cast<int>((g.m + BM - 1) / BM);
  p.band = kBand;
  p.wide_stores = (reinterpret_cast<uintptr_t>(g.c) & 31u) == 0;
  // A bf16 weight's tiles go to CTA pairs (half the operand bytes per SM and flop, two accumulator sets), in the width
  // that choose_pair_width picks.  Of a quantized weight's, 256-wide ones feed the tensor core better per shared-memory
  // byte and are taken when there are enough for the SMs; 128-wide ones keep a second accumulator set so the epilogue
  // overlaps the next tile.  CAIFQ_UMMA_BN overrides.
  const int mode = wmode_of(w, g.compute_dtype);
  const char *forced = std::getenv("CAIFQ_UMMA_BN");
  int bn = 128;
  bool pair = false;
  if (mode == W_BF16)
  {
    p.bn = pairs_enabled(mode) ? choose_pair_width(p.num_m_tiles, p.n_total, pair_count_umma()) : 0;
    if (forced != nullptr && p.bn != 0)
    {
      p.bn = std::atoi(forced) & ~31;
      p.bn = p.bn < 64 ? 64 : (p.bn > 256 ? 256 : p.bn);
    }
    pair = p.bn != 0;
    bn = pair ? p.bn : 128;
  }
  else
  {
    pair = pairs_enabled(mode) && (p.n_total % 256) == 0 &&
           static_cast<int64_t>(p.num_m_tiles) * (p.n_total / 256) >= pair_count_umma();
    bn = (pair || ((p.n_total % 256) == 0 &&
                   static_cast<int64_t>(p.num_m_tiles) * (p.n_total / 256) >= sm_count_umma()))
             ? 256
             : 128;
    if (forced != nullptr)
    {
      const int v = std::atoi(forced);
      if (v == 128 || (v == 256 && (p.n_total % 256) == 0))
      {
        bn = v;
      }
    }
    if (mode == W_I4S && !(pair && bn == 256))
    {
      bn = 128;   // a single CTA has 128-wide tiles only in the two-plane mode
    }
    pair = pair && bn == 256;
  }
  p.num_n_tiles = (p.n_total + bn - 1) / bn;

  CUtensorMap map_a;
  CUtensorMap map_b;
  int rc = make_map_bf16(&map_a, g.a, static_cast<uint64_t>(p.k_total), static_cast<uint64_t>(g.m), BM_SUB);
  if (rc != CAIFQ_OK)
  {
    return rc;
  }
  if (mode == W_BF16)
  {
    // the [out, in] weight itself: forward boxes are 64 k x 128 n rows, backward 64 n x 64 k rows
    rc = make_map_bf16(&map_b, w.codes, static_cast<uint64_t>(w.in_dim), static_cast<uint64_t>(w.out_dim),
                       g.backward ? BK : (pair ? bn / 2 : bn));
    if (rc != CAIFQ_OK)
    {
      return rc;
    }
  }
  else
  {
    map_b = map_a;
  }
  CUtensorMap map_h = map_a;
  CUtensorMap map_l = map_b;
  p.c_scale = (mode == W_BF16) ? g.c_scale : nullptr;
  if (g.lora_lhs != nullptr && g.lora_rhs != nullptr)
  {
    rc = make_map_bf16(&map_h, g.lora_lhs, 64, static_cast<uint64_t>(g.m), BM_SUB);
    if (rc != CAIFQ_OK)
    {
      return rc;
    }
    p.lora_rhs = static_cast<const uint8_t *>(g.lora_rhs);
    if (mode == W_BF16)
    {
      // the padded factor as a copy source: [N, 64] (forward, boxes of 64 k x the CTA's rows) or
      // [64, N] (backward, boxes of 64 n x 64 k), like the weight itself
      rc = g.backward ? make_map_bf16(&map_l, g.lora_rhs, static_cast<uint64_t>(p.n_total), 64, BK)
                      : make_map_bf16(&map_l, g.lora_rhs, 64, static_cast<uint64_t>(p.n_total),
                                      pair ? bn / 2 : bn);
      if (rc != CAIFQ_OK)
      {
        return rc;
      }
    }
  }
#define CAIFQ_UMMA_PAIR_CASE(MODE)                                                                      \
  if (mode == MODE && pair)                                                                \
  {                                                                                                     \
    return g.backward ? launch_inst<MODE, true, 256, false, true>(map_a, map_b, map_h, map_l, p, NoGroupTable{}, s)   \
                      : launch_inst<MODE, false, 256, false, true>(map_a, map_b, map_h, map_l, p, NoGroupTable{}, s); \
  }
  CAIFQ_UMMA_PAIR_CASE(W_I8)
  CAIFQ_UMMA_PAIR_CASE(W_I4)
  CAIFQ_UMMA_PAIR_CASE(W_BF16)
  CAIFQ_UMMA_PAIR_CASE(W_I4S)
#undef CAIFQ_UMMA_PAIR_CASE
#define CAIFQ_UMMA_CASE(MODE)                                                        \
  if (mode == MODE && bn == 128)                                                     \
  {                                                                                  \
    return g.backward ? launch_inst<MODE, true, 128, false>(map_a, map_b, map_h, map_l, p, NoGroupTable{}, s)   \
                      : launch_inst<MODE, false, 128, false>(map_a, map_b, map_h, map_l, p, NoGroupTable{}, s); \
  }                                                                                  \
  if (mode == MODE && bn == 256)                                                     \
  {                                                                                  \
    return g.backward ? launch_inst<MODE, true, 256, false>(map_a, map_b, map_h, map_l, p, NoGroupTable{}, s)   \
                      : launch_inst<MODE, false, 256, false>(map_a, map_b, map_h, map_l, p, NoGroupTable{}, s); \
  }
  CAIFQ_UMMA_CASE(W_I8)
  CAIFQ_UMMA_CASE(W_I4)
#undef CAIFQ_UMMA_CASE
  if (mode == W_BF16)
  {
    return g.backward ? launch_inst<W_BF16, true, 128, false>(map_a, map_b, map_h, map_l, p, NoGroupTable{}, s)
                      : launch_inst<W_BF16, false, 128, false>(map_a, map_b, map_h, map_l, p, NoGroupTable{}, s);
  }
  if (mode == W_I4S)   // two operand planes: 128-wide tiles only
  {
    return g.backward ? launch_inst<W_I4S, true, 128, false>(map_a, map_b, map_h, map_l, p, NoGroupTable{}, s)
                      : launch_inst<W_I4S, false, 128, false>(map_a, map_b, map_h, map_l, p, NoGroupTable{}, s);
  }
  set_error("frozen linear (umma): unsupported weight storage %d", w.storage);
  return CAIFQ_ERR_UNSUPPORTED;
}

// ------------------------------------------------------------------ grouped (frozen experts)
bool umma_grouped_supported(const GroupedLinearArgs &g)
{
  if (g.num_experts < 1 || g.weights == nullptr || g.offsets == nullptr)
  {
    return false;
  }
  const caifq_weight &w0 = g.weights[0];
  if ((w0.storage != CAIFQ_I8 && w0.storage != CAIFQ_I4 && w0.storage != CAIFQ_BF16) ||
      ((g.backward ? w0.in_dim : w0.out_dim) % 128) != 0)
  {
    return false;
  }
  if (w0.storage == CAIFQ_BF16)
  {
    // bf16 experts (expanded copies) are fed by tile copies from ONE tensor map: their matrices must lie
    // stacked, expert e at e * out * in elements behind expert 0
    const size_t stride = static_cast<size_t>(w0.in_dim) * static_cast<size_t>(w0.out_dim) * 2;
    for (int e = 0; e < g.num_experts; ++e)
    {
      if (static_cast<const char *>(g.weights[e].codes) != static_cast<const char *>(w0.codes) + e * stride)
      {
        return false;
      }
    }
  }
  LinearArgs probe{};
  probe.w = w0;
  probe.backward = g.backward;
  probe.a = g.a;
  probe.a_dtype = g.a_dtype;
  probe.a_prescale = 1.0f;
  probe.m = 32;   // the row count of a single expert does not matter here
  probe.c = g.c;
  probe.c_dtype = g.c_dtype;
  probe.accumulate = g.accumulate;
  probe.compute_dtype = g.compute_dtype;
  if (!umma_supported(probe))
  {
    return false;
  }
  for (int e = 0; e < g.num_experts; ++e)
  {
    const caifq_weight &w = g.weights[e];
    if (w.storage != w0.storage || w.scheme != w0.scheme || w.group_size != w0.group_size || w.in_dim != w0.in_dim ||
        w.out_dim != w0.out_dim || (w.scales == nullptr) != (w0.scales == nullptr) ||
        (reinterpret_cast<uintptr_t>(w.codes) & 15u) != 0)
    {
      return false;
    }
  }
  return g.offsets[g.num_experts] > 0;
}

int launch_linear_umma_grouped(const GroupedLinearArgs &g, cudaStream_t s)
{
  const caifq_weight &w0 = g.weights[0];
  const int64_t total_rows = g.offsets[g.num_experts];
  UmmaParams p{};
  p.spin_limit = kSpinLimit;
  p.stall_bytes = 0;
  p.codes = nullptr;
  p.scales = nullptr;
  p.c = g.c;
  p.c_dtype = g.c_dtype;
  p.accumulate = g.accumulate ? 1 : 0;
  p.wide_stores = ((reinterpret_cast<uintptr_t>(g.c) | reinterpret_cast<uintptr_t>(g.sb_g_up) |
                    reinterpret_cast<uintptr_t>(g.sb_gate) | reinterpret_cast<uintptr_t>(g.sb_up)) & 31u) == 0;
  p.m = total_rows;
  p.n_total = g.backward ? w0.in_dim : w0.out_dim;
  p.k_total = g.backward ? w0.out_dim : w0.in_dim;
  p.in_dim = w0.in_dim;
  p.group_size = w0.group_size;
  p.groups_per_row = (w0.group_size > 0) ? w0.in_dim / w0.group_size : 0;
  if (g.backward && g.sb_gate != nullptr && g.sb_up != nullptr && g.sb_g_up != nullptr && g.c_dtype == CAIFQ_BF16 &&
      !g.accumulate)
  {
    p.sb_gate = g.sb_gate;
    p.sb_up = g.sb_up;
    p.sb_g_up = g.sb_g_up;
  }
  CUtensorMap map_a;
  int rc = make_map_bf16(&map_a, g.a, static_cast<uint64_t>(p.k_total), static_cast<uint64_t>(total_rows), BM_SUB);
  if (rc != CAIFQ_OK)
  {
    return rc;
  }
  const int mode = wmode_of(w0, g.compute_dtype);
  for (int first = 0; first < g.num_experts; first += MAX_GROUPS)
  {
    const int count = (g.num_experts - first < MAX_GROUPS) ? (g.num_experts - first) : MAX_GROUPS;
    GroupTable gt{};
    int tiles = 0;
    for (int e = 0; e < count; ++e)
    {
      gt.offsets[e] = g.offsets[first + e];
      gt.mtile_start[e] = tiles;
      tiles += (g.offsets[first + e + 1] - g.offsets[first + e] + BM - 1) / BM;
      gt.codes[e] = static_cast<const uint8_t *>(g.weights[first + e].codes);
      gt.scales[e] = g.weights[first + e].scales;
    }
    gt.offsets[count] = g.offsets[first + count];
    gt.mtile_start[count] = tiles;
    gt.num_groups = count;
    if (tiles == 0)
    {
      continue;
    }
    p.num_m_tiles = tiles;
    // (for the experts' shapes the wide tile measured 3 % faster with int4 too, unlike the square case)
    // (an accumulating epilogue reads the output first: with 128-wide tiles it overlaps the next tile)
    // (pairs keep two accumulator sets at 256 columns, so the accumulating epilogue and the two-plane mode
    // can have the wide tile there)
    if (mode == W_BF16)
    {
      // stacked bf16 experts: one map over [count * out, in]; pairs when the width allows, else 128-wide tiles
      // (a width that is a multiple of 128 only, like 1408, still takes 256-wide pair tiles: the last tile's upper
      // half is masked in the epilogue, 9 % of wasted MMAs against 62 -> 85 % tensor activity)
      const int wide_tiles = (p.n_total + 255) / 256;
      const bool wide = static_cast<int64_t>(tiles) * wide_tiles >= pair_count_umma() && pairs_enabled(mode);
      p.bn = 256;
      p.num_n_tiles = wide ? wide_tiles : p.n_total / 128;
      p.expert_rows = w0.out_dim;
      CUtensorMap map_b;
      rc = make_map_bf16(&map_b, g.weights[first].codes, static_cast<uint64_t>(w0.in_dim),
                         static_cast<uint64_t>(count) * static_cast<uint64_t>(w0.out_dim), g.backward ? BK : 128);
      if (rc != CAIFQ_OK)
      {
        return rc;
      }
      // second operand pair (dX of two projections that share their input: C = A.W + A2.W2 in one accumulation)
      CUtensorMap map_a2 = map_a;
      CUtensorMap map_b2 = map_b;
      p.dual_k = 0;
      if (g.weights2 != nullptr && g.a2 != nullptr)
      {
        rc = make_map_bf16(&map_a2, g.a2, static_cast<uint64_t>(p.k_total), static_cast<uint64_t>(total_rows), BM_SUB);
        if (rc == CAIFQ_OK)
        {
          rc = make_map_bf16(&map_b2, g.weights2[first].codes, static_cast<uint64_t>(w0.in_dim),
                             static_cast<uint64_t>(count) * static_cast<uint64_t>(w0.out_dim), g.backward ? BK : 128);
        }
        if (rc != CAIFQ_OK)
        {
          return rc;
        }
        p.dual_k = 1;
      }
      if (wide)
      {
        rc = g.backward ? launch_inst<W_BF16, true, 256, true, true>(map_a, map_b, map_a2, map_b2, p, gt, s)
                        : launch_inst<W_BF16, false, 256, true, true>(map_a, map_b, map_a2, map_b2, p, gt, s);
      }
      else
      {
        rc = g.backward ? launch_inst<W_BF16, true, 128, true>(map_a, map_b, map_a2, map_b2, p, gt, s)
                        : launch_inst<W_BF16, false, 128, true>(map_a, map_b, map_a2, map_b2, p, gt, s);
      }
      if (rc != CAIFQ_OK)
      {
        return rc;
      }
      continue;
    }
    const bool pair = pairs_enabled(mode) && (p.n_total % 256) == 0 &&
                      static_cast<int64_t>(tiles) * (p.n_total / 256) >= pair_count_umma();
    const int bn = (pair || (mode != W_I4S && !g.accumulate && (p.n_total % 256) == 0 &&
                             static_cast<int64_t>(tiles) * (p.n_total / 256) >= sm_count_umma()))
                       ? 256
                       : 128;
    p.num_n_tiles = p.n_total / bn;
#define CAIFQ_UMMA_GROUP_PAIR_CASE(MODE)                                                           \
  if (mode == MODE && pair)                                                                        \
  {                                                                                                \
    rc = g.backward ? launch_inst<MODE, true, 256, true, true>(map_a, map_a, map_a, map_a, p, gt, s)      \
                    : launch_inst<MODE, false, 256, true, true>(map_a, map_a, map_a, map_a, p, gt, s);    \
  }
    CAIFQ_UMMA_GROUP_PAIR_CASE(W_I8)
    CAIFQ_UMMA_GROUP_PAIR_CASE(W_I4)
    CAIFQ_UMMA_GROUP_PAIR_CASE(W_I4S)
#undef CAIFQ_UMMA_GROUP_PAIR_CASE
    if (pair)
    {
      if (rc != CAIFQ_OK)
      {
        return rc;
      }
      continue;
    }
#define CAIFQ_UMMA_GROUP_CASE(MODE)                                                              \
  if (mode == MODE && bn == 128)                                                                 \
  {                                                                                              \
    rc = g.backward ? launch_inst<MODE, true, 128, true>(map_a, map_a, map_a, map_a, p, gt, s)          \
                    : launch_inst<MODE, false, 128, true>(map_a, map_a, map_a, map_a, p, gt, s);        \
  }                                                                                              \
  if (mode == MODE && bn == 256)                                                                 \
  {                                                                                              \
    rc = g.backward ? launch_inst<MODE, true, 256, true>(map_a, map_a, map_a, map_a, p, gt, s)          \
                    : launch_inst<MODE, false, 256, true>(map_a, map_a, map_a, map_a, p, gt, s);        \
  }
    CAIFQ_UMMA_GROUP_CASE(W_I8)
    CAIFQ_UMMA_GROUP_CASE(W_I4)
#undef CAIFQ_UMMA_GROUP_CASE
    if (mode == W_I4S)
    {
      rc = g.backward ? launch_inst<W_I4S, true, 128, true>(map_a, map_a, map_a, map_a, p, gt, s)
                      : launch_inst<W_I4S, false, 128, true>(map_a, map_a, map_a, map_a, p, gt, s);
    }
    if (rc != CAIFQ_OK)
    {
      return rc;
    }
  }
  return CAIFQ_OK;
}

// ------------------------------------------------------------------ fused gate / up / SwiGLU
bool umma_swiglu_supported(const GroupedSwigluArgs &g)
{
  if (g.num_experts < 1 || g.gate == nullptr || g.up == nullptr || g.offsets == nullptr || g.dtype != CAIFQ_BF16)
  {
    return false;
  }
  GroupedLinearArgs probe{};
  probe.weights = g.gate;
  probe.num_experts = g.num_experts;
  probe.offsets = g.offsets;
  probe.backward = false;
  probe.a = g.x;
  probe.a_dtype = g.dtype;
  probe.c = g.gate_out;
  probe.c_dtype = g.dtype;
  probe.accumulate = false;
  probe.compute_dtype = g.compute_dtype;
  if (!umma_grouped_supported(probe))
  {
    return false;
  }
  probe.weights = g.up;
  probe.c = g.up_out;
  if (!umma_grouped_supported(probe))
  {
    return false;
  }
  const caifq_weight &w0 = g.gate[0];
  const caifq_weight &u0 = g.up[0];
  if (u0.storage != w0.storage || u0.scheme != w0.scheme || u0.group_size != w0.group_size ||
      u0.in_dim != w0.in_dim || u0.out_dim != w0.out_dim || (w0.out_dim % 64) != 0)
  {
    return false;
  }
  return (reinterpret_cast<uintptr_t>(g.hidden) & 15u) == 0 && (reinterpret_cast<uintptr_t>(g.up_out) & 15u) == 0;
}

int launch_linear_umma_swiglu(const GroupedSwigluArgs &g, cudaStream_t s)
{
  const caifq_weight &w0 = g.gate[0];
  const int64_t total_rows = g.offsets[g.num_experts];
  UmmaParams p{};
  p.spin_limit = kSpinLimit;
  p.stall_bytes = 0;
  p.c = g.gate_out;
  p.c_up = g.up_out;
  p.c_hidden = g.hidden;
  p.c_dtype = g.dtype;
  p.accumulate = 0;
  p.wide_stores = ((reinterpret_cast<uintptr_t>(g.gate_out) | reinterpret_cast<uintptr_t>(g.up_out) |
                    reinterpret_cast<uintptr_t>(g.hidden)) & 31u) == 0;
  p.m = total_rows;
  p.n_total = 2 * w0.out_dim;   // gate and up features side by side in every tile
  p.k_total = w0.in_dim;
  p.in_dim = w0.in_dim;
  p.group_size = w0.group_size;
  p.groups_per_row = (w0.group_size > 0) ? w0.in_dim / w0.group_size : 0;
  p.swiglu = 1;
  p.bn = 256;
  CUtensorMap map_a;
  int rc = make_map_bf16(&map_a, g.x, static_cast<uint64_t>(p.k_total), static_cast<uint64_t>(total_rows), BM_SUB);
  if (rc != CAIFQ_OK)
  {
    return rc;
  }
  const int mode = wmode_of(w0, g.compute_dtype);
  for (int first = 0; first < g.num_experts; first += MAX_GROUPS)
  {
    const int count = (g.num_experts - first < MAX_GROUPS) ? (g.num_experts - first) : MAX_GROUPS;
    GroupTable gt{};
    int tiles = 0;
    for (int e = 0; e < count; ++e)
    {
      gt.offsets[e] = g.offsets[first + e];
      gt.mtile_start[e] = tiles;
      tiles += (g.offsets[first + e + 1] - g.offsets[first + e] + BM - 1) / BM;
      gt.codes[e] = static_cast<const uint8_t *>(g.gate[first + e].codes);
      gt.scales[e] = g.gate[first + e].scales;
      gt.codes_up[e] = static_cast<const uint8_t *>(g.up[first + e].codes);
      gt.scales_up[e] = g.up[first + e].scales;
    }
    gt.offsets[count] = g.offsets[first + count];
    gt.mtile_start[count] = tiles;
    gt.num_groups = count;
    if (tiles == 0)
    {
      continue;
    }
    p.num_m_tiles = tiles;
    // 128 features of each projection per tile on a CTA pair, 64 on a single CTA
    const bool pair = pairs_enabled(mode) && (w0.out_dim % 128) == 0 &&
                      static_cast<int64_t>(tiles) * (w0.out_dim / 128) >= pair_count_umma();
    p.num_n_tiles = w0.out_dim / (pair ? 128 : 64);
    if (mode == W_BF16)
    {
      p.expert_rows = w0.out_dim;
      CUtensorMap map_g;
      CUtensorMap map_u;
      const uint64_t rows = static_cast<uint64_t>(count) * static_cast<uint64_t>(w0.out_dim);
      rc = make_map_bf16(&map_g, g.gate[first].codes, static_cast<uint64_t>(w0.in_dim), rows, pair ? 128 : 64);
      if (rc == CAIFQ_OK)
      {
        rc = make_map_bf16(&map_u, g.up[first].codes, static_cast<uint64_t>(w0.in_dim), rows, pair ? 128 : 64);
      }
      if (rc != CAIFQ_OK)
      {
        return rc;
      }
      rc = pair ? launch_inst<W_BF16, false, 256, true, true>(map_a, map_g, map_a, map_u, p, gt, s)
                : launch_inst<W_BF16, false, 128, true>(map_a, map_g, map_a, map_u, p, gt, s);
    }
    else if (pair)
    {
      if (mode == W_I8)
      {
        rc = launch_inst<W_I8, false, 256, true, true>(map_a, map_a, map_a, map_a, p, gt, s);
      }
      else if (mode == W_I4S)
      {
        rc = launch_inst<W_I4S, false, 256, true, true>(map_a, map_a, map_a, map_a, p, gt, s);
      }
      else
      {
        rc = launch_inst<W_I4, false, 256, true, true>(map_a, map_a, map_a, map_a, p, gt, s);
      }
    }
    else if (mode == W_I8)
    {
      rc = launch_inst<W_I8, false, 128, true>(map_a, map_a, map_a, map_a, p, gt, s);
    }
    else if (mode == W_I4S)
    {
      rc = launch_inst<W_I4S, false, 128, true>(map_a, map_a, map_a, map_a, p, gt, s);
    }
    else
    {
      rc = launch_inst<W_I4, false, 128, true>(map_a, map_a, map_a, map_a, p, gt, s);
    }
    if (rc != CAIFQ_OK)
    {
      return rc;
    }
  }
  return CAIFQ_OK;
}

}  // namespace caifq
