// What the tcgen05 kernels share: mbarrier waits, tile copies, tensor-core instructions and descriptors in inline PTX,
// and the conversions of quantized codes to bf16 operands.
#pragma once

#include <cuda.h>

#include "common.cuh"

namespace caifq
{

namespace
{

constexpr uint32_t kSpinLimit = 1u << 22;       // polls of one wait before it gives up (tens of ms)
constexpr uint32_t kSpinLimitTest = 1u << 12;   // the same for the self-test of the give-up path

enum WMode
{
  W_I8 = 0,
  W_I4 = 1,
  W_BF16 = 2,
  // int4 for fp32 compute: scale * code (exact in fp32) goes to the tensor core as two bf16 terms,
  // hi = bf16(w) and lo = bf16(w - hi), in two operand planes; hi + lo equals w to 2^-17 relative
  W_I4S = 3
};

__host__ __device__ constexpr int planes_of(int wmode) { return wmode == W_I4S ? 2 : 1; }

// ------------------------------------------------------------------ PTX helpers
__device__ __forceinline__ uint32_t smem_u32(const void *p)
{
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count)
{
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes)
{
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar)
{
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

// Bounded wait.  A wait that runs out raises the CTA's abort word and the device flag; from then on
// every wait of the CTA returns at once, so the roles run through the rest of their loops without
// spinning (on garbage: the results are wrong and the host sees the flag) and the kernel ends within
// about one limit, TMEM released.
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity)
{
  uint32_t done;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(done)
      : "r"(bar), "r"(parity)
      : "memory");
  return done != 0;
}

__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile uint32_t *abort_word, uint32_t limit,
                                          unsigned int *device_flag)
{
  // A barrier that is already complete costs one poll and nothing else: the abort word is looked at only
  // once a wait actually has to wait (reading it before every poll cost 12 % of the kernel's throughput).
  if (mbar_try(bar, parity))
  {
    return true;
  }
  if (*abort_word != 0u)
  {
    return false;
  }
  for (uint32_t spin = 0; spin < limit; ++spin)
  {
    if (mbar_try(bar, parity))
    {
      return true;
    }
    if ((spin & 1023u) == 1023u && *abort_word != 0u)
    {
      return false;
    }
  }
  *abort_word = 1u;
  atomicExch(device_flag, 1u);
  return false;
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *map, int c0, int c1, uint32_t bar)
{
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
          dst),
      "l"(map), "r"(c0), "r"(c1), "r"(bar)
      : "memory");
}

// ---- two-CTA (cluster) forms
__device__ __forceinline__ uint32_t cluster_ctarank()
{
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}

// the shared::cluster address of `addr` (a shared::cta address of this CTA) in the CTA of rank `rank`
__device__ __forceinline__ uint32_t map_to_cta(uint32_t addr, uint32_t rank)
{
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}

__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_bar)
{
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}

__device__ __forceinline__ uint32_t ld_shared_cluster(uint32_t cluster_addr)
{
  uint32_t v;
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(cluster_addr) : "memory");
  return v;
}

__device__ __forceinline__ void cluster_sync_all()
{
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// A tile load of this CTA's own shared memory whose bytes are counted on a barrier of the pair's leader CTA
// (`cluster_bar`, a shared::cluster address).  No multicast: every CTA fetches its own tile.
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap *map, int c0, int c1,
                                                 uint32_t cluster_bar)
{
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], "
      "[%4];" ::"r"(dst),
      "l"(map), "r"(c0), "r"(c1), "r"(cluster_bar)
      : "memory");
}

__device__ __forceinline__ void fence_proxy_async()
{
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void tc_fence_before()
{
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}

__device__ __forceinline__ void tc_fence_after()
{
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                          uint32_t accumulate)
{
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// one MMA of 256 rows over the CTA pair: each CTA's shared memory holds its 128 rows of A and its half of B
// at the same offsets, the accumulator rows land in each CTA's own tensor memory
__device__ __forceinline__ void umma_bf16_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                               uint32_t accumulate)
{
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

__device__ __forceinline__ bool elect_one()
{
  uint32_t pred;
  asm volatile(
      "{\n\t.reg .pred P;\n\t"
      "elect.sync _|P, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, P;\n\t}"
      : "=r"(pred));
  return pred != 0;
}

// arrive on an mbarrier once every MMA issued so far by this thread has finished
__device__ __forceinline__ void umma_commit(uint32_t bar)
{
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// the same for the pair's MMAs; the arrival goes to the barrier at this offset in both CTAs
__device__ __forceinline__ void umma_commit_pair(uint32_t bar)
{
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
      "h"(static_cast<uint16_t>(3))
      : "memory");
}

// the same, arriving on a barrier of the issuing CTA only
__device__ __forceinline__ void umma_commit_pair_local(uint32_t bar)
{
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16])
{
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32])
{
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,"
      "%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}

__device__ __forceinline__ void tmem_ld_wait()
{
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// Shared-memory matrix descriptor (sm_100): start address, leading / stride
// byte offsets in 16-byte units, descriptor version 1, 128-byte swizzle.
__device__ __forceinline__ uint64_t make_desc(uint32_t saddr, uint32_t lbo_bytes, uint32_t sbo_bytes)
{
  uint64_t d = 0;
  d |= static_cast<uint64_t>((saddr & 0x3FFFFu) >> 4);
  d |= static_cast<uint64_t>((lbo_bytes >> 4) & 0x3FFFu) << 16;
  d |= static_cast<uint64_t>((sbo_bytes >> 4) & 0x3FFFu) << 32;
  d |= 1ull << 46;  // version
  d |= 2ull << 61;  // SWIZZLE_128B
  return d;
}

// Instruction descriptor, kind::f16: fp32 accumulate, bf16 x bf16, A K-major,
// B K-major (forward) or MN-major (backward), N = 128, M = 128.
__host__ __device__ constexpr uint32_t make_idesc(bool b_mn_major, int BN, int M = 128)
{
  return (1u << 4)                          // D format f32
         | (1u << 7)                        // A format bf16
         | (1u << 10)                       // B format bf16
         | (0u << 15)                       // A major: K
         | ((b_mn_major ? 1u : 0u) << 16)   // B major
         | (static_cast<uint32_t>(BN >> 3) << 17) | (static_cast<uint32_t>(M >> 4) << 24);
}

__device__ __forceinline__ uint32_t lop3_and_or(uint32_t a, uint32_t b, uint32_t c)
{
  uint32_t d;
  asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}

__device__ __forceinline__ uint32_t sub_bf16x2(uint32_t a, uint32_t b)
{
  uint32_t d;
  asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}

__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi)
{
  uint32_t d;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
  return d;
}

// four int8 codes (one 32-bit word, memory order) -> two bf16x2 registers, exact
__device__ __forceinline__ void int8x4_to_bf16(uint32_t w, uint32_t &p01, uint32_t &p23)
{
  const uint32_t a = __byte_perm(w, 0u, 0x4140);  // [b0, 0, b1, 0]
  const uint32_t b = __byte_perm(w, 0u, 0x4342);  // [b2, 0, b3, 0]
  // low 7 bits dropped into the mantissa of 128.0; the sign bit selects 128.0 or 256.0 to subtract
  p01 = sub_bf16x2(lop3_and_or(a, 0x007F007Fu, 0x43004300u), lop3_and_or(a, 0x00800080u, 0x43004300u));
  p23 = sub_bf16x2(lop3_and_or(b, 0x007F007Fu, 0x43004300u), lop3_and_or(b, 0x00800080u, 0x43004300u));
}

__device__ __forceinline__ uint32_t mul_bf16x2(uint32_t a, uint32_t b)
{
  uint32_t d;
  asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}

// Eight int4 codes (one 32-bit word, memory order) times a scale -> four bf16x2 registers, for bf16
// compute.  The codes become exact bf16 integers with logic ops (the offset-binary nibble dropped into
// the mantissa of 128.0, then 136 subtracted: exact) and are multiplied by the group scale rounded to
// bf16, one rounding.  The reference's dequantize-then-cast forms scale * code in fp32 and rounds once;
// the two differ by the bf16 rounding of the fp16 scale (2^-9 relative), far inside the bf16 bound, and
// the conversion takes 17 instructions per eight weights instead of 31: the int4 launches are bound by
// this conversion, not by the tensor core.  One asm block: a loop of conversions and tensor-memory stores takes
// 53.2 us, with the same steps as C++ and single instructions 62.4 (4096 -> 14336, 96 tokens, 20.9 -> 20.8 us;
// 4096 -> 4096, 48 tokens, 11.2 -> 11.1).
__device__ __forceinline__ void int4x8_to_bf16(uint32_t w, uint32_t scale2, uint32_t (&out)[4])
{
  // e: u0 u2 u4 u6 (u = q + 8), d: u1 u3 u5 u7; t, v: in element order; 0x43: the high byte of bf16 128.0 .. 143.0
  asm("{\n\t.reg .b32 e, d, t, v;\n\t"
      "lop3.b32 e, %4, 0x0F0F0F0F, 0x08080808, 0x6A;\n\t"
      "shr.u32 d, %4, 4;\n\t"
      "lop3.b32 d, d, 0x0F0F0F0F, 0x08080808, 0x6A;\n\t"
      "prmt.b32 t, e, d, 0x5140;\n\t"
      "prmt.b32 v, e, d, 0x7362;\n\t"
      "prmt.b32 %0, t, 0x43434343, 0x4140;\n\t"
      "prmt.b32 %1, t, 0x43434343, 0x4342;\n\t"
      "prmt.b32 %2, v, 0x43434343, 0x4140;\n\t"
      "prmt.b32 %3, v, 0x43434343, 0x4342;\n\t"
      "sub.rn.bf16x2 %0, %0, %6;\n\t"
      "sub.rn.bf16x2 %1, %1, %6;\n\t"
      "sub.rn.bf16x2 %2, %2, %6;\n\t"
      "sub.rn.bf16x2 %3, %3, %6;\n\t"
      "mul.rn.bf16x2 %0, %0, %5;\n\t"
      "mul.rn.bf16x2 %1, %1, %5;\n\t"
      "mul.rn.bf16x2 %2, %2, %5;\n\t"
      "mul.rn.bf16x2 %3, %3, %5;\n\t}"
      : "=&r"(out[0]), "=&r"(out[1]), "=&r"(out[2]), "=&r"(out[3])
      : "r"(w), "r"(scale2), "r"(0x43084308u));
}

// the same eight codes as two bf16 terms of scale * code: hi = bf16(w), lo = bf16(w - hi)
__device__ __forceinline__ void int4x8_to_bf16_split(uint32_t w, float scale, uint32_t (&hi)[4], uint32_t (&lo)[4])
{
  const uint32_t ev = (w & 0x0F0F0F0Fu) ^ 0x08080808u;
  const uint32_t od = ((w >> 4) & 0x0F0F0F0Fu) ^ 0x08080808u;
  const float base = 8388616.0f;   // 2^23 + 8
#pragma unroll
  for (int j = 0; j < 4; ++j)
  {
    const float a = __fmul_rn(__uint_as_float(__byte_perm(ev, 0x4B000000u, 0x7440 + j)) - base, scale);
    const float b = __fmul_rn(__uint_as_float(__byte_perm(od, 0x4B000000u, 0x7440 + j)) - base, scale);
    const uint32_t h = pack_bf16x2(a, b);
    hi[j] = h;
    lo[j] = pack_bf16x2(a - __uint_as_float(h << 16), b - __uint_as_float(h & 0xFFFF0000u));
  }
}

// ------------------------------------------------------------------ host side
inline int wmode_of(const caifq_weight &w, int compute_dtype)
{
  if (w.storage == CAIFQ_I8)
  {
    return W_I8;
  }
  if (w.storage == CAIFQ_I4)
  {
    return (compute_dtype == CAIFQ_F32) ? W_I4S : W_I4;
  }
  return W_BF16;
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline EncodeTiledFn encode_fn()
{
  static EncodeTiledFn fn = nullptr;
  if (fn == nullptr)
  {
    void *ptr = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
    {
      fn = reinterpret_cast<EncodeTiledFn>(ptr);
    }
  }
  return fn;
}

// 2-D bf16 tensor map: `inner` contiguous elements per row, `outer` rows, box of 64 x box_rows, 128-byte swizzle.
inline int make_map_bf16(CUtensorMap *map, const void *base, uint64_t inner, uint64_t outer, uint32_t box_rows)
{
  EncodeTiledFn fn = encode_fn();
  if (fn == nullptr)
  {
    set_error("frozen linear (umma): cuTensorMapEncodeTiled is not available from the driver");
    return CAIFQ_ERR_CUDA;
  }
  const cuuint64_t dims[2] = {inner, outer};
  const cuuint64_t strides[1] = {inner * 2};
  const cuuint32_t box[2] = {64, box_rows};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(base), dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS)
  {
    set_error("frozen linear (umma): cuTensorMapEncodeTiled failed with %d", static_cast<int>(r));
    return CAIFQ_ERR_CUDA;
  }
  return CAIFQ_OK;
}

}  // namespace

}  // namespace caifq
