// Frozen-linear forward for some tens to a few hundred tokens, and for experts that see a few rows each:
//
//   C[m, out] = A[m, in] . W_deq[out, in]^T  (+ C)      (ForwardImpl, src/caif_device_frozen_linear.cpp:381-524;
//                                                        the expert loop, src/caif_device_moe_layer.cpp:534-557)
//
// Such a call would like to be bound by reading the packed codes once (4096 -> 14336 int4: 4.5 us of HBM).  What bounds it
// is turning them into bf16 (59 M weights at 2.2 instructions, half of them on pipes that take one every two cycles: 6.7 us
// in a loop of nothing else) and handing 32 stages over to the MMAs and back: of 20.8 us at 96 tokens 19.1 are left without
// the conversion, 17.0 without scales and stores too.  From 200 tokens on the tensor core needs as long.  The many-token
// kernel makes the tokens the rows of the tile: 256 of them however few there are, two 16-KB operand tiles in shared memory,
// mostly zeros, and one 4-KB tile of codes in flight.
// Here the roles are swapped: 128 weight rows are the M of the MMA and the tokens its N, 16 to 256 in steps of 16.  The
// converted weight goes to tensor memory as the A operand, which leaves shared memory's bandwidth to the codes and the
// activations (256 tokens: 50 us with A in shared memory, 40 with it here).
// 4096 -> 14336 int4, us a call, many-token kernel (converting) / this one: 17 tokens 42 / 20, 96 tokens 42 / 21, 256 tokens
// 44 / 29, 512 tokens 79 / 52; 4096 -> 4096: 38 / 11, 38 / 13, 41 / 19, 41 / 27; 64 experts of 2048 x 1408, 16 tokens top-6, three
// products: 249 / 121.
//
// One persistent CTA per SM, 19 warps, over tiles of 128 weight rows x up to 256 tokens:
//   warps 0, 18 TMA producers for the activation tiles
//   warp 1      TMEM allocation, MMA issue (one elected lane)
//   warps 2-17  codes: two teams of eight warps take alternate stages of 128 k, so one converts while the other's stage
//               is multiplied; a warp owns 32 rows x 64 k of a stage, copies its pieces into its own ring (cp.async,
//               64 bytes a row and unit, no barrier), converts them to bf16 and stores its part of the operand to tensor
//               memory (a lane is a weight row there).  The same warps drain the accumulators, after they have converted
//               their first stage of the next tile; a token's 32 rows leave as one contiguous store.
// Few row tiles (narrow layers) split k over the CTAs of a cluster; their partial tiles meet through distributed shared
// memory in rank order: no scratch, no atomics, the same bits every time.
// The codes' copies start before the kernel waits for the previous one in the stream (programmatic dependent launch); so
// do the first places' conversions.
//
// Operands and roundings are those of the many-token kernel: int8 codes exact in bf16 with the scale in the epilogue,
// int4 times its group scale rounded to bf16, or as two bf16 terms for fp32 compute.
//
// Every wait is bounded; a wait that runs out sets a flag that the host can read and lets the kernel finish (with wrong
// numbers) instead of hanging.
#include <atomic>

#include "umma.cuh"

namespace caifq
{

__device__ unsigned int g_stream_timeout_flag = 0;

// Reads and clears the flag (1 = some bounded wait ran out since the last call; -1 = query failed).
int take_stream_timeout_flag()
{
  unsigned int v = 0;
  const unsigned int zero = 0;
  if (cudaMemcpyFromSymbol(&v, g_stream_timeout_flag, sizeof(v)) != cudaSuccess ||
      (v != 0 && cudaMemcpyToSymbol(g_stream_timeout_flag, &zero, sizeof(zero)) != cudaSuccess))
  {
    return -1;
  }
  return v ? 1 : 0;
}

namespace
{

constexpr int ROWS = 128;            // weight rows of a tile
constexpr int TOKENS = 256;          // most tokens of a tile (N of one MMA)
constexpr int KB = 64;               // k of an operand tile: one 128-byte swizzle span of bf16
// Tensor memory: accumulators in columns 0..255 (two sets of 128 tokens, or one of 256), then two stages of the weight
// operand: 32 columns per 64 k and plane (a lane is a weight row, a column two bf16 values).
constexpr uint32_t A_COLUMN0 = 256;
constexpr uint32_t SUB_COLUMNS = 32;
constexpr uint32_t PLANE_COLUMNS = 2 * SUB_COLUMNS;   // of a stage (128 k)
constexpr int WARPS = 19;
constexpr int CODE_WARP0 = 2;
constexpr int CODE_WARPS = 16;
constexpr int SECOND_COPY_WARP = CODE_WARP0 + CODE_WARPS;
constexpr uint32_t UNIT_BYTES = 32 * 64;    // a warp's 32 rows x 64 bytes of codes
constexpr int MAX_B = 6;                    // activation stages (128 k each) in flight
constexpr int DONE = 8;                     // ring of "stage multiplied" barriers
constexpr int TMEM_COLUMNS = 512;
constexpr uint32_t SMEM_LIMIT = 226u * 1024u;
constexpr uint32_t SCALES_LIMIT = 40u * 1024u;   // more would cost the activations their places
// Three tiles of tokens.  Set when 768 tokens of 4096 -> 14336 took 94 us and 1024 took 124, the many-token kernel 119 and
// 120; it is still ahead at the line for every layer measured.  us at 768 tokens here, at 769 expanded / converted there:
// 4096 -> 14336 int4 78, 108 / 111; 14336 -> 4096 84, 107 / 118; 4096 -> 4096 29, 38 / 39; int8 79, 110 / 127; 85, 104 / 116;
// 29, 37 / 38.
constexpr int kStreamMostTokens = 768;

struct StreamEntry
{
  const uint8_t *codes;
  const void *scales;
  void *c;               // [.., n_total]; row 0 is packed row 0
  int row0;              // first packed row
  int rows;
  int tile_start;        // tiles of the entries before this one
};

constexpr int MAX_ENTRIES = 160;

template <int N>
struct StreamTable
{
  StreamEntry e[N];
  int count;
};

struct StreamParams
{
  int c_dtype;
  int accumulate;
  int n_total;           // features of every entry
  int k_total;
  uint32_t row_bytes;    // packed bytes of a weight row
  GroupOf group_of;      // int4
  int groups_per_row;
  int group_size;
  uint32_t scales_at;    // their place in shared memory
  uint32_t scale_bytes;  // int4: of a tile's 128 rows, where they are copied to shared memory; 0 = read from global memory
  int num_tiles;
  int splits;            // CTAs of a cluster (k ranges)
  int box;               // tokens per activation copy
  int tile_tokens;       // most tokens of a tile
  int b_stages;          // places for activations: of 128 k, or of 64 k where `halves` is set
  int halves;
  int acc_bufs;          // accumulator sets: 2 of 128 columns, or 1 of 256
  int depth;             // units in flight per code warp: 2 or 3
  uint32_t b_sub_bytes;  // 64 k of the activations
  uint32_t b_stage_bytes;
  uint32_t spin_limit;
  uint32_t stall_bytes;  // self-test only: bytes the first activation tile announces but never receives
};

// A tile, as the warps of its CTA read it from shared memory
struct StreamTile
{
  const uint8_t *codes;      // of its first weight row
  const void *scales;        // int4: of its first weight row; int8: the weight's one scale, or null
  void *c;                   // element (first token, first weight row) of the result
  int token0;                // first packed row
  int tokens;
};
static_assert(sizeof(StreamTile) == 32, "one 32-byte record");

template <bool IS_I4, int N>
__device__ __forceinline__ StreamTile locate(const StreamParams &p, const StreamTable<N> &t, int tile)
{
  int lo = 0;
  if (N > 1)
  {
    int hi = t.count;   // tile_start[lo] <= tile < tile_start[hi]
    while (hi - lo > 1)
    {
      const int mid = (lo + hi) >> 1;
      if (t.e[mid].tile_start <= tile)
      {
        lo = mid;
      }
      else
      {
        hi = mid;
      }
    }
  }
  const StreamEntry &e = t.e[lo];
  const int local = tile - e.tile_start;
  const int chunks = (e.rows + p.tile_tokens - 1) / p.tile_tokens;   // neighbours share the codes, through L2
  const int chunk = local % chunks;
  const int64_t row = static_cast<int64_t>(local / chunks) * ROWS;
  StreamTile w;
  w.codes = e.codes + row * p.row_bytes;
  w.scales = IS_I4 ? static_cast<const uint16_t *>(e.scales) + row * p.groups_per_row : e.scales;
  w.token0 = e.row0 + chunk * p.tile_tokens;
  w.tokens = min(p.tile_tokens, e.rows - chunk * p.tile_tokens);
  w.c = static_cast<char *>(e.c) + (static_cast<int64_t>(w.token0) * p.n_total + row) * (p.c_dtype == CAIFQ_F32 ? 4 : 2);
  return w;
}

__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src)
{
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

__device__ __forceinline__ uint4 lds128(uint32_t addr)
{
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
  return v;
}

// 16 words of every lane into 16 columns of the warp's quarter of tensor memory
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16])
{
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}

__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// D += A . B^T with A in tensor memory
__device__ __forceinline__ void umma_bf16_tmem(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc,
                                               uint32_t accumulate)
{
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem_d),
      "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

template <int WMODE, int N, bool HALVES>
__global__ void __launch_bounds__(WARPS * 32, 1)
linear_stream_kernel(const __grid_constant__ CUtensorMap map_b, const __grid_constant__ StreamParams p,
                     const __grid_constant__ StreamTable<N> table)
{
  constexpr bool IS_I4 = (WMODE == W_I4 || WMODE == W_I4S);
  constexpr int PLANES = planes_of(WMODE);
  constexpr int UNIT_STAGES = IS_I4 ? 2 : 1;          // stages of one team in a unit of codes
  constexpr uint32_t STAGE_CODES = IS_I4 ? 64u : 128u;   // bytes of a row per stage
  constexpr uint32_t STAGE_COLUMNS = PLANE_COLUMNS * PLANES;
  constexpr uint32_t PLACES = 256u / STAGE_COLUMNS;   // stages of the weight operand: 4, or 2 of two planes
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t bars[4 + DONE + 2 * MAX_B + 4 + 2];
  __shared__ uint64_t drain_bar;   // give-up path only: the MMAs issued so far have completed
  __shared__ uint32_t tmem_base_slot;
  __shared__ uint32_t cta_abort;   // a wait of this CTA has run out

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t b_place_bytes = HALVES ? p.b_sub_bytes : p.b_stage_bytes;
  auto b_addr = [&](uint32_t s) { return smem_base + s * b_place_bytes; };
  const uint32_t ring_base = smem_base + static_cast<uint32_t>(p.b_stages) * b_place_bytes;
  const uint32_t bar0 = smem_u32(bars);
  const uint32_t tiles_base = ring_base + static_cast<uint32_t>(CODE_WARPS * p.depth) * UNIT_BYTES;
  const StreamTile *tiles = reinterpret_cast<const StreamTile *>(smem_raw + (tiles_base - smem_u32(smem_raw)));
  auto a_full = [&](uint32_t s) { return bar0 + s * 8u; };
  auto done = [&](uint32_t g) { return bar0 + (4u + g % DONE) * 8u; };
  auto done_parity = [&](uint32_t g) { return (g / DONE) & 1u; };
  auto b_full = [&](uint32_t s) { return bar0 + (4u + DONE + s) * 8u; };
  auto b_empty = [&](uint32_t s) { return bar0 + (4u + DONE + MAX_B + s) * 8u; };   // halves only
  auto acc_full = [&](int a) { return bar0 + static_cast<uint32_t>(4 + DONE + 2 * MAX_B + a) * 8u; };
  auto acc_empty = [&](int a) { return bar0 + static_cast<uint32_t>(4 + DONE + 2 * MAX_B + 2 + a) * 8u; };
  auto sc_full = [&](int i) { return bar0 + static_cast<uint32_t>(4 + DONE + 2 * MAX_B + 4 + (i & 1)) * 8u; };
  // int4: the scales of tile i (its rows' are contiguous), in one of two places after the tile records
  auto scales_at = [&](int i) { return p.scales_at + smem_base + static_cast<uint32_t>(i & 1) * p.scale_bytes; };
  // (the warps' arrivals and the copies' bytes have separate barriers: after a wait that ran out the warps run on, and an
  // arrival beyond the count of a barrier that still expects bytes is a fault)
  volatile uint32_t *abort_word = &cta_abort;
  auto wait = [&](uint32_t bar, uint32_t parity)
  { return mbar_wait(bar, parity, abort_word, p.spin_limit, &g_stream_timeout_flag); };

  const int rank = p.splits > 1 ? static_cast<int>(cluster_ctarank()) : 0;
  const int worker = static_cast<int>(blockIdx.x) / p.splits;
  const int workers = static_cast<int>(gridDim.x) / p.splits;
  // this CTA's tiles, looked up once: a search of the table by every warp at every tile took longer than a small tile
  const int num_tiles = (p.num_tiles - worker + workers - 1) / workers;
  for (int i = static_cast<int>(threadIdx.x); i < num_tiles; i += WARPS * 32)
  {
    const_cast<StreamTile *>(tiles)[i] = locate<IS_I4>(p, table, worker + i * workers);
  }
  if (threadIdx.x == 0)
  {
    cta_abort = 0u;
    mbar_init(smem_u32(&drain_bar), 1);
    for (uint32_t s = 0; s < PLACES; ++s)
    {
      mbar_init(a_full(s), 8);
    }
    for (uint32_t s = 0; s < DONE; ++s)
    {
      mbar_init(done(s), 1);
    }
    for (uint32_t s = 0; s < MAX_B; ++s)
    {
      mbar_init(b_full(s), 1);
      mbar_init(b_empty(s), 1);
    }
    for (int a = 0; a < 2; ++a)
    {
      mbar_init(acc_full(a), 1);
      mbar_init(sc_full(a), 1);
      mbar_init(acc_empty(a), CODE_WARPS);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1)
  {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_slot)),
                 "r"(TMEM_COLUMNS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_slot;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

  // this CTA's range of k, in whole stages
  const int all_kb = p.k_total / KB;
  const int all_stages = (all_kb + 1) / 2;
  const int st_begin = (all_stages * rank) / p.splits;
  const int stages = (all_stages * (rank + 1)) / p.splits - st_begin;
  const int num_kb = min(all_kb - 2 * st_begin, 2 * stages);

  if (warp == 0 || warp == SECOND_COPY_WARP)
  {
    // ------------------------------------------------------- activation tiles
    // Two threads, each copies the tile of one 64-k half of every stage: one that waited, announced the bytes and issued
    // both copies needed 700 cycles a stage and kept the MMAs waiting.
    // HALVES: tiles of more than 128 tokens (64 KB a stage) have places of 64 k, freed one by one: two places of 128 k
    // left the MMAs waiting for 570 of 1380 cycles a stage (256 tokens: 33 us, now 30).  Half h has every other place.
    // Fewer tokens keep whole stages: there the one thread that issues the MMAs is the limit, and a wait and a commit more
    // a stage cost 7 %.
    const int half = warp == 0 ? 0 : 1;
    const uint32_t own = static_cast<uint32_t>(p.b_stages) / 2u;
    auto produce = [&]()
    {
      asm volatile("griddepcontrol.wait;" ::: "memory");
      uint32_t s = 0;
      uint32_t g = 0;
      uint32_t n = 0;   // halves copied so far
      for (int tile = 0; tile < num_tiles; ++tile)
      {
        const StreamTile w = tiles[tile];
        const int boxes = (w.tokens + p.box - 1) / p.box;
        const uint32_t box_bytes = static_cast<uint32_t>(p.box) * 128u;
        for (int st = 0; st < stages; ++st, ++g)
        {
          const int subs = min(2, num_kb - 2 * st);
          if (HALVES)
          {
            if (half < subs)
            {
              const uint32_t at = 2u * (n % own) + static_cast<uint32_t>(half);
              if (n >= own && !wait(b_empty(at), (n / own - 1u) & 1u))
              {
                return;
              }
              mbar_expect_tx(b_full(at), static_cast<uint32_t>(boxes) * box_bytes + (g == 0 && half == 0 ? p.stall_bytes : 0u));
              for (int b = 0; b < boxes; ++b)
              {
                tma_load_2d(b_addr(at) + static_cast<uint32_t>(b) * box_bytes, &map_b, (2 * (st_begin + st) + half) * KB,
                            w.token0 + b * p.box, b_full(at));
              }
              ++n;
            }
            continue;
          }
          // (A stage of one half is multiplied without the second thread, which must then not wait for it either: the
          // stages may be DONE ahead of it by the time it looks, and the parity it waits for past.)
          if (half < subs)
          {
            // the place of the stage b_stages before this one: it must have been multiplied
            if (g >= static_cast<uint32_t>(p.b_stages))
            {
              const uint32_t old = g - static_cast<uint32_t>(p.b_stages);
              if (!wait(done(old), done_parity(old)))
              {
                return;   // nothing new is started once a wait has run out
              }
            }
            if (half == 0)
            {
              mbar_expect_tx(b_full(s), static_cast<uint32_t>(subs * boxes) * box_bytes + (g == 0 ? p.stall_bytes : 0u));
            }
            const uint32_t to = b_addr(s) + static_cast<uint32_t>(half) * p.b_sub_bytes;
            for (int b = 0; b < boxes; ++b)
            {
              tma_load_2d(to + static_cast<uint32_t>(b) * box_bytes, &map_b, (2 * (st_begin + st) + half) * KB,
                          w.token0 + b * p.box, b_full(s));
            }
          }
          if (++s == static_cast<uint32_t>(p.b_stages))
          {
            s = 0;
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
    // ------------------------------------------------------------- MMA issuer
    // One lane, and as few instructions as it takes: this warp shares its scheduler with four that convert without a
    // pause, so every instruction here waits its turn (with a barrier per 64 k, and an election and a warp barrier per
    // stage, a stage took 1100 cycles, of which the tensor core was at work 330).
    // It stops at the first wait that runs out: a barrier that still expects bytes must not be armed again, and the producer
    // arms one only after the stage before it in that place has been committed here.
    auto multiply = [&]()
    {
      uint32_t g = 0;    // stages multiplied so far
      uint32_t sb = 0, b_par = 0;
      uint32_t halves[2] = {0, 0};   // multiplied so far
      const uint32_t own = static_cast<uint32_t>(p.b_stages) / 2u;
      int acc = 0;
      uint32_t acc_par = 0;
      const uint64_t bdesc_base = make_desc(smem_base, 16, 1024);
      auto copy_scales = [&](int tile)
      {
        // (not once a wait has run out: the place's barrier may still expect bytes)
        if (IS_I4 && p.scale_bytes != 0u && tile < num_tiles && *abort_word == 0u)
        {
          mbar_expect_tx(sc_full(tile), p.scale_bytes);
          asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                           scales_at(tile)),
                       "l"(tiles[tile].scales), "r"(p.scale_bytes), "r"(sc_full(tile))
                       : "memory");
        }
      };
      copy_scales(0);
      // (the activations come after the previous kernel: the limit of a wait must not run while that one does)
      asm volatile("griddepcontrol.wait;" ::: "memory");
      for (int tile = 0; tile < num_tiles; ++tile)
      {
        // (everything of the tile before this one has been converted, so its scales' place is free)
        copy_scales(tile + 1);
        const uint32_t idesc = make_idesc(false, (tiles[tile].tokens + 15) & ~15, ROWS);
        const uint32_t d = tmem_base + static_cast<uint32_t>(acc * 128);
        if (!wait(acc_empty(acc), acc_par ^ 1u))
        {
          return;
        }
        uint32_t accumulate = 0;
        for (int st = 0; st < stages; ++st, ++g)
        {
          const uint32_t a0 = tmem_base + A_COLUMN0 + (g % PLACES) * STAGE_COLUMNS;
          uint64_t bdesc0 = bdesc_base + static_cast<uint64_t>((sb * p.b_stage_bytes) >> 4);
          if ((!HALVES && !wait(b_full(sb), b_par)) || !wait(a_full(g % PLACES), (g / PLACES) & 1u))
          {
            return;
          }
          tc_fence_after();
#pragma unroll
          for (int h = 0; h < 2; ++h)
          {
            if (h == 0 || 2 * st + 1 < num_kb)
            {
              uint32_t at = 0;
              if (HALVES)
              {
                at = 2u * (halves[h] % own) + static_cast<uint32_t>(h);
                if (!wait(b_full(at), (halves[h] / own) & 1u))
                {
                  return;
                }
                tc_fence_after();
                ++halves[h];
                bdesc0 = bdesc_base + static_cast<uint64_t>((b_addr(at) - smem_base - (h ? p.b_sub_bytes : 0u)) >> 4);
              }
#pragma unroll
              for (int k16 = 0; k16 < KB / 16; ++k16)
              {
                const uint32_t a = a0 + static_cast<uint32_t>(h) * SUB_COLUMNS + static_cast<uint32_t>(k16 * 8);
                const uint64_t bdesc = bdesc0 + static_cast<uint64_t>(h ? p.b_sub_bytes >> 4 : 0u) + static_cast<uint64_t>(k16 * 2);
                umma_bf16_tmem(d, a, bdesc, idesc, (h == 0 && k16 == 0) ? accumulate : 1u);
                if (PLANES == 2)
                {
                  umma_bf16_tmem(d, a + PLANE_COLUMNS, bdesc, idesc, 1u);
                }
              }
              if (HALVES)
              {
                umma_commit(b_empty(at));
              }
            }
          }
          umma_commit(done(g));
          accumulate = 1;
          if (++sb == static_cast<uint32_t>(p.b_stages))
          {
            sb = 0;
            b_par ^= 1u;
          }
        }
        umma_commit(acc_full(acc));
        if (++acc == p.acc_bufs)
        {
          acc = 0;
          acc_par ^= 1u;
        }
      }
    };
    if (elect_one())
    {
      multiply();
    }
    __syncwarp();
  }
  else
  {
    // ------------------------------------------------------ codes and epilogue
    const int cw = warp - CODE_WARP0;
    const int team = cw >> 3;
    const int half = (cw >> 2) & 1;              // which 64 k of a stage
    const int wq = warp & 3;                     // this warp's rows: 32 wq .. 32 wq + 31 of the tile, and TMEM lanes
    const uint32_t ring = ring_base + static_cast<uint32_t>(cw * p.depth) * UNIT_BYTES;
    // drains the accumulators of a tile: this warp's TMEM lanes (the 32 of its rows), every fourth run of 16 tokens
    int acc = 0;
    uint32_t acc_par = 0;
    auto epilogue = [&](int tile)
    {
      const StreamTile w = tiles[tile];
      const float out_scale =
          (WMODE == W_I8 && w.scales != nullptr) ? __ldg(static_cast<const float *>(w.scales)) : 1.0f;
      const int column = wq * 32 + lane;
      wait(acc_full(acc), acc_par);
      tc_fence_after();
      for (int t0 = 16 * (((cw >> 2) + tile) & 3); t0 < w.tokens; t0 += 64)   // (few tokens: the warps take turns)
      {
        uint32_t r[16];
        tmem_ld16(tmem_base + (static_cast<uint32_t>(wq * 32) << 16) + static_cast<uint32_t>(acc * 128 + t0), r);
        tmem_ld_wait();
        const int64_t at = static_cast<int64_t>(t0) * p.n_total + column;
        const int count = min(16, w.tokens - t0);
        if (p.splits > 1)
        {
          // partial sums [token][128 rows], over the activation tiles and rings: everything in them has been used
#pragma unroll
          for (int j = 0; j < 16; ++j)
          {
            if (j < count)
            {
              asm volatile("st.shared.u32 [%0], %1;" ::"r"(smem_base + static_cast<uint32_t>((t0 + j) * ROWS + column) * 4u),
                           "r"(r[j])
                           : "memory");
            }
          }
        }
        else if (p.c_dtype == CAIFQ_F32 && !p.accumulate)
        {
          float *dst = static_cast<float *>(w.c) + at;
#pragma unroll
          for (int j = 0; j < 16; ++j)
          {
            if (j < count)
            {
              dst[static_cast<int64_t>(j) * p.n_total] = __uint_as_float(r[j]) * out_scale;
            }
          }
        }
        else if (p.c_dtype == CAIFQ_BF16 && !p.accumulate)
        {
          __nv_bfloat16 *dst = static_cast<__nv_bfloat16 *>(w.c) + at;
#pragma unroll
          for (int j = 0; j < 16; ++j)
          {
            if (j < count)
            {
              dst[static_cast<int64_t>(j) * p.n_total] = __float2bfloat16(__uint_as_float(r[j]) * out_scale);
            }
          }
        }
        else
        {
#pragma unroll
          for (int j = 0; j < 16; ++j)
          {
            if (j < count)
            {
              const int64_t i = at + static_cast<int64_t>(j) * p.n_total;
              float v = __uint_as_float(r[j]) * out_scale;
              if (p.accumulate)
              {
                v = round_through_rt(v, p.c_dtype) + load_as_float(w.c, i, p.c_dtype);
              }
              store_from_float(w.c, i, p.c_dtype, v);
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0)
      {
        mbar_arrive(acc_empty(acc));
      }
      if (++acc == p.acc_bufs)
      {
        acc = 0;
        acc_par ^= 1u;
      }
    };
    // copies: a lane takes one 16-byte piece of rows lane / 4, + 8, ...; pieces XOR the row pair, so that eight lanes
    // reading eight rows' same piece hit different banks
    const uint32_t piece = static_cast<uint32_t>(lane & 3);
    const uint32_t copy_row = static_cast<uint32_t>(lane >> 2);
    // a unit is 64 bytes of every row: this warp's half of UNIT_STAGES stages of its team (every other stage)
    const uint32_t piece_stage = 2u * (IS_I4 ? piece >> 1 : 0u);
    const uint32_t piece_byte = piece_stage * STAGE_CODES + static_cast<uint32_t>(half) * (STAGE_CODES / 2) +
                                (IS_I4 ? piece & 1u : piece) * 16u;
    // stages of this team in tile i: the first of them, and their number in units
    auto first_stage = [&](int i) { return team ^ ((i * stages) & 1); };
    auto units_of = [&](int i) { return ((stages - first_stage(i) + 1) / 2 + UNIT_STAGES - 1) / UNIT_STAGES; };
    int f_tile = -1;
    int f_left = 0;          // units of the tile being copied that are still to come
    bool f_last = false;     // this lane's piece of the last of them exists
    const uint8_t *f_src = nullptr;
    const size_t rows8 = static_cast<size_t>(8) * p.row_bytes;
    const uint32_t copy_dst = copy_row * 64u + ((piece ^ ((copy_row >> 1) & 3u)) << 4);
    auto fetch = [&](uint32_t slot)
    {
      while (f_left == 0 && f_tile + 1 < num_tiles)   // (a team may have no stage in a tile of one stage)
      {
        ++f_tile;
        const int first = first_stage(f_tile);
        f_left = units_of(f_tile);
        const int last = 2 * UNIT_STAGES * (f_left - 1);
        const uint32_t at = static_cast<uint32_t>(st_begin + first) * STAGE_CODES + piece_byte;
        f_last = f_left > 0 && at + static_cast<uint32_t>(last) * STAGE_CODES < p.row_bytes &&
                 first + last + static_cast<int>(piece_stage) < stages;
        f_src = tiles[f_tile].codes + static_cast<size_t>(wq * 32 + static_cast<int>(copy_row)) * p.row_bytes + at;
        if (IS_I4 && p.scale_bytes == 0u)
        {
          // the scales of this lane's row are on their way to L2 before the first of them is used
          const char *sc = static_cast<const char *>(tiles[f_tile].scales) +
                           static_cast<int64_t>(wq * 32 + lane) * p.groups_per_row * 2;
          for (int b = 0; b < p.groups_per_row * 2; b += 128)
          {
            asm volatile("prefetch.global.L2 [%0];" ::"l"(sc + b));
          }
        }
      }
      if (f_left > 1 || (f_left == 1 && f_last))
      {
        const uint8_t *src = f_src;
#pragma unroll
        for (uint32_t i = 0; i < 4; ++i, src += rows8)
        {
          cp_async16(slot + copy_dst + i * 512u, src);
        }
      }
      f_src += 2 * UNIT_STAGES * STAGE_CODES;
      f_left = f_left > 0 ? f_left - 1 : 0;
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    const uint32_t ring_end = ring + static_cast<uint32_t>(p.depth) * UNIT_BYTES;
    for (uint32_t slot = ring; slot != ring_end; slot += UNIT_BYTES)
    {
      fetch(slot);
    }
    uint32_t slot = ring;
    uint32_t g_before = 0;   // stages of the tiles before this one
    const uint32_t ring_sw = static_cast<uint32_t>((lane >> 1) & 3);
    const uint32_t dst = tmem_base + (static_cast<uint32_t>(wq * 32) << 16) + A_COLUMN0 +
                         static_cast<uint32_t>(half) * SUB_COLUMNS;
    // int4: the scales of a unit's 32-code pieces.  A lane owns a row, so reading them from global memory touches 32 lines
    // a time: they are copied to shared memory a tile ahead, unless the rows are too long for that (14336 -> 4096,
    // 17 tokens: 23.4 us without, 21.9 with; two operand planes, 4096 -> 14336, 512 tokens: 114 and 109).
    const bool pairs = (p.group_size % KB) == 0;   // both pieces of a stage have one scale
    auto load_scales = [&](int tile, int first, int unit, uint16_t (&sc)[4])
    {
      const uint16_t *global =
          static_cast<const uint16_t *>(tiles[tile].scales) + static_cast<int64_t>(wq * 32 + lane) * p.groups_per_row;
      const uint32_t shared = scales_at(tile) + static_cast<uint32_t>((wq * 32 + lane) * p.groups_per_row) * 2u;
#pragma unroll
      for (int i = 0; i < 4; ++i)
      {
        if ((i & 1) && pairs)
        {
          sc[i] = sc[i - 1];
        }
        else
        {
          const int k = ((st_begin + first + 2 * (UNIT_STAGES * unit + (i >> 1))) * 2 + half) * KB + (i & 1) * 32;
          const uint32_t group = p.group_of(static_cast<uint32_t>(min(k, p.k_total - 1)));
          if (p.scale_bytes != 0u)
          {
            asm volatile("ld.shared.u16 %0, [%1];" : "=h"(sc[i]) : "r"(shared + group * 2u));
          }
          else
          {
            sc[i] = __ldg(global + group);
          }
        }
      }
    };
    uint16_t next_sc[4];   // read from global memory: loaded while the unit before is converted
    if (IS_I4 && p.scale_bytes == 0u && num_tiles > 0)
    {
      load_scales(0, first_stage(0), 0, next_sc);
    }
    int undrained = -1;   // a tile whose accumulators still wait
    // Before the first wait on what follows from an MMA, and before anything is written: the kernel before this one has
    // ended.  Until then its time would count against the wait's limit, and it may read what is written here.
    bool released = false;
    auto after_previous = [&]()
    {
      if (!released)
      {
        asm volatile("griddepcontrol.wait;" ::: "memory");
        released = true;
      }
    };
    // one trip more than there are tiles, to drain the last one
    for (int tile = 0; tile <= num_tiles; ++tile, g_before += static_cast<uint32_t>(stages))
    {
      const int first = first_stage(tile);
      const int units = tile < num_tiles ? units_of(tile) : 0;
      for (int unit = 0; unit == 0 || unit < units; ++unit)
      {
        // (with one accumulator set before anything of the next tile, which could not be multiplied)
        if (undrained >= 0 && (unit >= 1 || units <= 1 || p.acc_bufs == 1))
        {
          after_previous();
          epilogue(undrained);
          undrained = -1;
        }
        if (unit >= units)
        {
          break;
        }
        if (p.depth == 3)
        {
          asm volatile("cp.async.wait_group 2;" ::: "memory");
        }
        else
        {
          asm volatile("cp.async.wait_group 1;" ::: "memory");
        }
        __syncwarp();   // every lane's copies have landed
        uint4 v[4];
#pragma unroll
        for (uint32_t i = 0; i < 4; ++i)
        {
          v[i] = lds128(slot + static_cast<uint32_t>(lane) * 64u + ((i ^ ring_sw) << 4));
        }
        float sc[IS_I4 ? 4 : 1];
        if constexpr (IS_I4)
        {
          if (p.scale_bytes != 0u)
          {
            if (unit == 0)
            {
              if (tile > 0)   // (the first tile's scales are on their way at once)
              {
                after_previous();
              }
              wait(sc_full(tile), static_cast<uint32_t>(tile >> 1) & 1u);
            }
            load_scales(tile, first, unit, next_sc);
          }
#pragma unroll
          for (int i = 0; i < 4; ++i)
          {
            sc[i] = __half2float(__ushort_as_half(next_sc[i]));
          }
        }
        __syncwarp();   // the slot has been read by every lane: refill it
        fetch(slot);
        slot += UNIT_BYTES;
        slot = slot == ring_end ? ring : slot;
        if (IS_I4 && p.scale_bytes == 0u)
        {
          if (unit + 1 < units)
          {
            load_scales(tile, first, unit + 1, next_sc);
          }
          else if (tile + 1 < num_tiles)
          {
            load_scales(tile + 1, first_stage(tile + 1), 0, next_sc);
          }
        }
#pragma unroll
        for (int u = 0; u < UNIT_STAGES; ++u)
        {
          const int stage = first + 2 * (UNIT_STAGES * unit + u);
          if (stage < stages)
          {
            const uint32_t g = g_before + static_cast<uint32_t>(stage);
            const uint32_t place = dst + (g % PLACES) * STAGE_COLUMNS;
            bool placed = false;
#pragma unroll
            for (int c = 0; c < 2; ++c)
            {
              uint32_t o[16];
              uint32_t l[16];
#pragma unroll
              for (int q = 0; q < 4; ++q)
              {
                if constexpr (WMODE == W_I8)
                {
                  const uint4 x = v[2 * c + (q >> 1)];
                  int8x4_to_bf16((q & 1) ? x.z : x.x, o[4 * q + 0], o[4 * q + 1]);
                  int8x4_to_bf16((q & 1) ? x.w : x.y, o[4 * q + 2], o[4 * q + 3]);
                }
                else
                {
                  const uint4 x = v[2 * u + c];
                  const uint32_t word = q == 0 ? x.x : (q == 1 ? x.y : (q == 2 ? x.z : x.w));
                  uint32_t o4[4];
                  uint32_t l4[4] = {0, 0, 0, 0};
                  if constexpr (WMODE == W_I4S)
                  {
                    int4x8_to_bf16_split(word, sc[2 * u + c], o4, l4);
                  }
                  else
                  {
                    int4x8_to_bf16(word, pack_bf16x2(sc[2 * u + c], sc[2 * u + c]), o4);
                  }
#pragma unroll
                  for (int e = 0; e < 4; ++e)
                  {
                    o[4 * q + e] = o4[e];
                    l[4 * q + e] = l4[e];
                  }
                }
              }
              if (!placed)
              {
                placed = true;
                if (g >= PLACES)
                {
                  after_previous();
                  wait(done(g - PLACES), done_parity(g - PLACES));
                  tc_fence_after();
                }
              }
              // (the second half of an odd last stage is not multiplied: whatever it holds)
              tmem_st16(place + static_cast<uint32_t>(16 * c), o);
              if constexpr (WMODE == W_I4S)
              {
                tmem_st16(place + PLANE_COLUMNS + static_cast<uint32_t>(16 * c), l);
              }
            }
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0)
            {
              mbar_arrive(a_full(g % PLACES));
            }
          }
        }
      }
      undrained = tile;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
  }
  __syncwarp();

  // ---------------------------------------------------------------- k splits
  if (p.splits > 1)
  {
    cluster_sync_all();   // the partial tiles are complete (one tile per cluster)
    const StreamTile w = tiles[0];
    const int t_begin = (w.tokens * rank) / p.splits;
    const int t_end = (w.tokens * (rank + 1)) / p.splits;
    const float out_scale =
        (WMODE == W_I8 && w.scales != nullptr) ? __ldg(static_cast<const float *>(w.scales)) : 1.0f;
    for (int i = static_cast<int>(threadIdx.x); i < (t_end - t_begin) * ROWS; i += WARPS * 32)
    {
      const int token = t_begin + (i >> 7);
      const uint32_t local = smem_base + static_cast<uint32_t>(token * ROWS + (i & 127)) * 4u;
      float v = 0.0f;
      for (int r = 0; r < p.splits; ++r)
      {
        v += __uint_as_float(ld_shared_cluster(map_to_cta(local, static_cast<uint32_t>(r))));
      }
      v *= out_scale;
      const int64_t at = static_cast<int64_t>(token) * p.n_total + (i & 127);
      if (p.accumulate)
      {
        v = round_through_rt(v, p.c_dtype) + load_as_float(w.c, at, p.c_dtype);
      }
      store_from_float(w.c, at, p.c_dtype, v);
    }
    cluster_sync_all();   // nobody's shared memory is read after this
  }

  // ---------------------------------------------------------------- teardown
  const uint32_t gave_up = *abort_word;
  if (gave_up != 0u && warp == 0 && lane == 0)
  {
    // activation tiles that were started may still be on their way: give them time to land before the CTA's shared
    // memory goes back
    for (int i = 0; i < 64; ++i)
    {
      __nanosleep(2000);
    }
  }
  if (gave_up != 0u && warp == 1)
  {
    // MMAs issued after the give-up may still run: tensor memory is released only after they have completed
    if (elect_one())
    {
      umma_commit(smem_u32(&drain_bar));
    }
    __syncwarp();
    bool done = false;
    for (uint32_t spin = 0; spin < p.spin_limit && !done; ++spin)
    {
      done = mbar_try(smem_u32(&drain_bar), 0u);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1)
  {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLUMNS) : "memory");
  }
}

// ------------------------------------------------------------------ host side
int stream_ctas() { return persistent_ctas("CAIFQ_UMMA_CTAS"); }

// A CTA keeps a record of each of its tiles in shared memory.  With at most 1024 of them (32 KB) two places for
// activations and the codes in flight always fit beside them; one CTA of a large layer (a host that leaves this library few
// SMs) may have more, and is the many-token kernel's.
constexpr int64_t kMostTilesPerCta = 1024;

bool records_fit(int64_t tiles) { return tiles <= kMostTilesPerCta * stream_ctas(); }

// What shares the memory of an SM: codes in flight and activation tiles.
bool choose_depths(StreamParams &p, uint32_t &smem)
{
  const int ctas = stream_ctas();
  const uint32_t per_cta = static_cast<uint32_t>((p.num_tiles + ctas - 1) / ctas);
  const uint32_t records = per_cta * static_cast<uint32_t>(sizeof(StreamTile));
  const uint32_t scales = p.scale_bytes * (per_cta > 1 ? 2u : 1u);
  if (scales > SCALES_LIMIT)
  {
    p.scale_bytes = 0;
  }
  p.halves = p.acc_bufs == 1 ? 1 : 0;   // more than 128 tokens
  const uint32_t place = p.halves ? p.b_sub_bytes : p.b_stage_bytes;
  const int want = (p.halves || place <= 16384) ? 4 : (place <= 32768 ? 3 : 2);
  for (int least = want; least >= 2; --least)
  {
    for (int depth : {3, 2})   // units of codes per warp
    {
      const uint32_t fixed = static_cast<uint32_t>(CODE_WARPS * depth) * UNIT_BYTES + ((records + 15u) & ~15u) + (p.scale_bytes != 0u ? scales : 0u) + 1024u;
      if (fixed + static_cast<uint32_t>(least) * place <= SMEM_LIMIT)
      {
        int fit = static_cast<int>((SMEM_LIMIT - fixed) / place);
        fit = p.halves ? fit & ~1 : fit;
        p.depth = depth;
        p.b_stages = fit < MAX_B ? fit : MAX_B;
        smem = fixed + static_cast<uint32_t>(p.b_stages) * place;
        p.scales_at = static_cast<uint32_t>(p.b_stages) * place +
                      static_cast<uint32_t>(CODE_WARPS * depth) * UNIT_BYTES + ((records + 15u) & ~15u);
        return true;
      }
    }
  }
  return false;
}

// Clusters of `size` CTAs (one per SM) that run at the same time: GPCs are not multiples of every size, and a few of their
// SMs may be missing, so this is asked for, once per kernel and device.  A query that fails counts as none for its call.
template <typename K>
int resident_clusters(K kernel, std::atomic<int> &known, int size)
{
  int n = known.load(std::memory_order_relaxed);
  if (n == 0)
  {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(static_cast<unsigned>(size));
    cfg.blockDim = dim3(WARPS * 32);
    cfg.dynamicSmemBytes = SMEM_LIMIT;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = static_cast<unsigned>(size);
    attr.val.clusterDim.y = 1;
    attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess || n < 1)
    {
      cudaGetLastError();
      return 0;
    }
    known.store(n, std::memory_order_relaxed);
  }
  return n;
}

template <int WMODE, int N, bool HALVES>
int launch_stream_inst(const CUtensorMap &map_b, StreamParams &p, const StreamTable<N> &table, uint32_t smem,
                       bool dependent, cudaStream_t s)
{
  auto kernel = linear_stream_kernel<WMODE, N, HALVES>;
  static std::atomic<bool> configured[kMaxDevices];
  int dev = 0;
  CAIFQ_CHECK_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices)
  {
    set_error("frozen linear (stream): device ordinal %d out of range", dev);
    return CAIFQ_ERR_UNSUPPORTED;
  }
  if (!configured[dev].load(std::memory_order_acquire))
  {
    CAIFQ_CHECK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(SMEM_LIMIT)));
    configured[dev].store(true, std::memory_order_release);
  }
  if (N == 1)
  {
    // k is split where all clusters run at once, with at least four 64-k tiles for every CTA and room for the partial tile
    // in shared memory
    static std::atomic<int> clusters[kMaxDevices][9];   // by size; of this kernel
    const int num_kb = p.k_total / KB;
    for (int c : {8, 4, 3, 2})
    {
      if (p.num_tiles * c <= stream_ctas() && num_kb >= 4 * c && p.num_tiles <= resident_clusters(kernel, clusters[dev][c], c) &&
          p.b_sub_bytes * 4u + 32u + p.scale_bytes + 1024u <= smem)
      {
        p.splits = c;
        break;
      }
    }
  }
  cudaLaunchConfig_t cfg{};
  const int most = stream_ctas();
  cfg.gridDim = dim3(static_cast<unsigned>(p.splits > 1 ? p.num_tiles * p.splits : (p.num_tiles < most ? p.num_tiles : most)));
  cfg.blockDim = dim3(WARPS * 32);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = static_cast<unsigned>(p.splits);
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = dependent ? 2 : 1;
  CAIFQ_CHECK_CUDA(cudaLaunchKernelEx(&cfg, kernel, map_b, p, table));
  return CAIFQ_OK;
}

template <int N>
int launch_stream(int mode, const CUtensorMap &map_b, StreamParams &p, const StreamTable<N> &table, uint32_t smem,
                  cudaStream_t s)
{
  // codes written just ahead in this stream by one of the library's own calls: a plain launch orders the early copies
  // behind that kernel
  const bool dependent = dependent_launches() && !take_codes_written(s);
  switch (mode)
  {
    case W_I8:
      return p.halves ? launch_stream_inst<W_I8, N, true>(map_b, p, table, smem, dependent, s)
                      : launch_stream_inst<W_I8, N, false>(map_b, p, table, smem, dependent, s);
    case W_I4:
      return p.halves ? launch_stream_inst<W_I4, N, true>(map_b, p, table, smem, dependent, s)
                      : launch_stream_inst<W_I4, N, false>(map_b, p, table, smem, dependent, s);
    default:
      return launch_stream_inst<W_I4S, N, false>(map_b, p, table, smem, dependent, s);
  }
}

bool weight_streams(const caifq_weight &w, int compute_dtype)
{
  if ((w.out_dim % ROWS) != 0 || (w.in_dim % KB) != 0 || (reinterpret_cast<uintptr_t>(w.codes) & 15u) != 0 ||
      (compute_dtype != CAIFQ_BF16 && compute_dtype != CAIFQ_F32))
  {
    return false;
  }
  if (w.storage == CAIFQ_I8)
  {
    return w.scales == nullptr || w.scheme == CAIFQ_PER_TENSOR;
  }
  return w.storage == CAIFQ_I4 && w.scales != nullptr && w.group_size > 0 && (w.group_size % 32) == 0 &&
         (w.in_dim % w.group_size) == 0;
}

// (two operand planes leave tensor memory for two accumulator sets of 128 tokens)
int tile_tokens(int mode) { return mode == W_I4S ? 128 : TOKENS; }

StreamParams common_params(const caifq_weight &w, int mode, int c_dtype, bool accumulate, int most_rows,
                           bool scales_aligned, bool grouped)
{
  StreamParams p{};
  p.c_dtype = c_dtype;
  p.accumulate = accumulate ? 1 : 0;
  p.n_total = w.out_dim;
  p.k_total = w.in_dim;
  p.row_bytes = static_cast<uint32_t>(w.storage == CAIFQ_I4 ? w.in_dim / 2 : w.in_dim);
  p.group_of = GroupOf::make(w.group_size > 0 ? w.group_size : 1);
  p.group_size = w.group_size;
  p.groups_per_row = w.storage == CAIFQ_I4 ? w.in_dim / w.group_size : 0;
  p.scale_bytes = scales_aligned ? static_cast<uint32_t>(p.groups_per_row) * (ROWS * 2u) : 0u;
  p.splits = 1;
  p.tile_tokens = tile_tokens(mode);
  const int most_tokens = most_rows < p.tile_tokens ? most_rows : p.tile_tokens;
  p.acc_bufs = most_tokens <= 128 ? 2 : 1;
  // one copy a tile where the tiles are alike, little over-fetch where experts have a row here and hundreds there
  p.box = (!grouped || most_tokens <= 32) ? (most_tokens + 15) & ~15 : (most_tokens <= 128 ? 32 : 64);
  p.b_sub_bytes = static_cast<uint32_t>((most_tokens + p.box - 1) / p.box * p.box) * 128u;
  p.b_stage_bytes = 2u * p.b_sub_bytes;
  p.spin_limit = kSpinLimit;
  p.stall_bytes = 0;
  if (take_umma_stall())
  {
    // self-test of the give-up path: the first activation tile announces 16 bytes that never arrive
    p.spin_limit = kSpinLimitTest;
    p.stall_bytes = 16;
  }
  return p;
}

}  // namespace

bool stream_supported(const LinearArgs &g)
{
  const int most = stream_ctas();
  if (g.compute_dtype == CAIFQ_F32 && g.w.storage == CAIFQ_I4 && g.m > 128 &&
      (g.w.out_dim / ROWS) * ((g.m + 127) / 128) > most)
  {
    // Two operand planes leave room for 128 tokens a tile, so every 128 tokens convert again.  That pays while all tiles
    // run at once (4096 -> 4096, 512 tokens: 43 us against 71), not from the second wave on (-> 14336, 256: 78 against 62).
    return false;
  }
  return !g.backward && g.a_dtype == CAIFQ_BF16 && g.a_prescale == 1.0f && g.m >= 17 && g.m <= kStreamMostTokens &&
         g.lora_lhs == nullptr && g.num_peers == 0 && g.num_more == 0 && is_float_dtype(g.c_dtype) &&
         (reinterpret_cast<uintptr_t>(g.a) & 15u) == 0 && weight_streams(g.w, g.compute_dtype) &&
         records_fit((g.w.out_dim / ROWS) * ((g.m + 127) / 128));
}

int launch_linear_stream(const LinearArgs &g, cudaStream_t s)
{
  const caifq_weight &w = g.w;
  const int mode = wmode_of(w, g.compute_dtype);
  const int m = static_cast<int>(g.m);
  StreamParams p = common_params(w, mode, g.c_dtype, g.accumulate, m, (reinterpret_cast<uintptr_t>(w.scales) & 15u) == 0, false);
  StreamTable<1> table{};
  table.count = 1;
  table.e[0].codes = static_cast<const uint8_t *>(w.codes);
  table.e[0].scales = w.scales;
  table.e[0].c = g.c;
  table.e[0].row0 = 0;
  table.e[0].rows = m;
  table.e[0].tile_start = 0;
  p.num_tiles = (w.out_dim / ROWS) * ((m + p.tile_tokens - 1) / p.tile_tokens);
  uint32_t smem = 0;
  if (!choose_depths(p, smem))
  {
    set_error("frozen linear (stream): no stage fits");
    return CAIFQ_ERR_UNSUPPORTED;
  }
  CUtensorMap map_b;
  const int rc = make_map_bf16(&map_b, g.a, static_cast<uint64_t>(w.in_dim), static_cast<uint64_t>(m),
                               static_cast<uint32_t>(p.box));
  if (rc != CAIFQ_OK)
  {
    return rc;
  }
  return launch_stream(mode, map_b, p, table, smem, s);
}

bool stream_grouped_supported(const GroupedStreamArgs &g)
{
  if (g.count < 1 || g.count > MAX_ENTRIES || g.total_rows < 1 || !is_float_dtype(g.c_dtype) ||
      (reinterpret_cast<uintptr_t>(g.a) & 15u) != 0)
  {
    return false;
  }
  const caifq_weight &w0 = g.weights[0];
  int64_t tiles = 0;
  for (int e = 0; e < g.count; ++e)
  {
    const caifq_weight &w = g.weights[e];
    if (!weight_streams(w, g.compute_dtype) || w.storage != w0.storage || w.in_dim != w0.in_dim ||
        w.out_dim != w0.out_dim || w.group_size != w0.group_size || (w.scales == nullptr) != (w0.scales == nullptr))
    {
      return false;
    }
    tiles += (w0.out_dim / ROWS) * ((static_cast<int64_t>(g.row_end[e]) - g.row_begin[e] + 127) / 128);
  }
  return records_fit(tiles);
}

int launch_linear_stream_grouped(const GroupedStreamArgs &g, cudaStream_t s)
{
  const caifq_weight &w0 = g.weights[0];
  const int mode = wmode_of(w0, g.compute_dtype);
  static thread_local StreamTable<MAX_ENTRIES> table;
  int most = 0;
  int tiles = 0;
  bool scales_aligned = true;
  table.count = 0;
  for (int e = 0; e < g.count; ++e)
  {
    const int rows = g.row_end[e] - g.row_begin[e];
    if (rows <= 0)
    {
      continue;
    }
    StreamEntry &t = table.e[table.count++];
    t.codes = static_cast<const uint8_t *>(g.weights[e].codes);
    t.scales = g.weights[e].scales;
    scales_aligned = scales_aligned && (reinterpret_cast<uintptr_t>(t.scales) & 15u) == 0;
    t.c = g.c[e];
    t.row0 = g.row_begin[e];
    t.rows = rows;
    t.tile_start = tiles;
    tiles += (w0.out_dim / ROWS) * ((rows + tile_tokens(mode) - 1) / tile_tokens(mode));
    most = rows > most ? rows : most;
  }
  if (tiles == 0)
  {
    return CAIFQ_OK;
  }
  StreamParams p = common_params(w0, mode, g.c_dtype, g.accumulate, most, scales_aligned, true);
  p.num_tiles = tiles;
  uint32_t smem = 0;
  if (!choose_depths(p, smem))
  {
    set_error("frozen experts (stream): no stage fits");
    return CAIFQ_ERR_UNSUPPORTED;
  }
  CUtensorMap map_b;
  const int rc = make_map_bf16(&map_b, g.a, static_cast<uint64_t>(w0.in_dim), static_cast<uint64_t>(g.total_rows),
                               static_cast<uint32_t>(p.box));
  if (rc != CAIFQ_OK)
  {
    return rc;
  }
  return launch_stream(mode, map_b, p, table, smem, s);
}

}  // namespace caifq
