// tcgen05 / TMA building blocks shared by the tensor-core kernels (16-bit GEMM and the exact-slice
// FP64 emulation): mbarrier waits bounded by the global timer, 2D TMA loads, UMMA descriptors for
// 128-byte-swizzled K-major tiles, tcgen05.mma/commit/ld wrappers, and the host-side tensor-map and
// instruction-descriptor encoders.
#pragma once
#include <cuda.h>

#include "ofrr_internal.cuh"

namespace ofrr {
namespace tc {

constexpr int BM = 128;
constexpr int BK = 64;  // one 128-byte swizzle row of 16-bit elements

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ uint64_t globaltimer() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// bounded wait (about 2 s); records code in *err and returns false on timeout
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, int* err, int code,
                                          uint64_t limit_ns = 2000000000ull) {
  if (mbar_try_wait(bar, parity)) return true;
  const uint64_t t0 = globaltimer();
  while (true) {
    if (mbar_try_wait(bar, parity)) return true;
    if (globaltimer() - t0 > limit_ns) {
      atomicCAS(err, 0, code);
      return false;
    }
  }
}
// mbar_wait by a whole warp, with one answer for its lanes, which leave it converged.  (Every lane polls and reads the
// timer by itself: near the limit one may give up while another sees the phase complete, and lanes that part there would
// wait for each other at the next warp-wide operation and at the CTA's barrier, for ever.)
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* bar, uint32_t parity, int* err, int code,
                                               uint64_t limit_ns = 2000000000ull) {
  return __all_sync(0xffffffffu, mbar_wait(bar, parity, err, code, limit_ns));
}

__device__ __forceinline__ void tma_load_2d(const CUtensorMap* map, uint64_t* bar, void* dst, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
          smem_u32(dst)),
      "l"((uint64_t)map), "r"(x), "r"(y), "r"(smem_u32(bar))
      : "memory");
}

// UMMA shared-memory descriptor of a K-major operand with 128-byte swizzle: bits 0-13 the start address in 16-byte
// units, 16-29 the leading byte offset (ignored here, 1), 32-45 the stride between 8-row groups (1024 B in 16-byte
// units), bit 46 the version, 61-63 the swizzle (2 = 128 bytes).  Only the low word varies, by the address.
constexpr uint32_t kDescLo = 1u << 16;
constexpr uint32_t kDescHi = (1024u >> 4) | (1u << 14) | (2u << 29);

// D (TMEM) += A B, both operands by their descriptors' low words (shared address >> 4).
// F8: E4M3 x E4M3 -> FP32 (kind::f8f6f4), K = 32 bytes per instruction like the 16-bit form
template <bool F8>
__device__ __forceinline__ void umma_lo(uint32_t tmem_d, uint32_t a_lo, uint32_t b_lo, uint32_t idesc,
                                        uint32_t accumulate) {
  if (F8)
    asm volatile(
        "{\n .reg .pred p;\n .reg .b64 a, b;\n mov.b64 a, {%1, %5};\n mov.b64 b, {%2, %5};\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], a, b, %3, p;\n}\n" ::"r"(tmem_d),
        "r"(a_lo | kDescLo), "r"(b_lo | kDescLo), "r"(idesc), "r"(accumulate), "r"(kDescHi)
        : "memory");
  else
    asm volatile(
        "{\n .reg .pred p;\n .reg .b64 a, b;\n mov.b64 a, {%1, %5};\n mov.b64 b, {%2, %5};\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, p;\n}\n" ::"r"(tmem_d),
        "r"(a_lo | kDescLo), "r"(b_lo | kDescLo), "r"(idesc), "r"(accumulate), "r"(kDescHi)
        : "memory");
}
// A from TMEM (128 lanes x 8 columns of two 16-bit values per K = 16), B by its descriptor's low word (shared address
// >> 4)
__device__ __forceinline__ void umma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint32_t b_lo, uint32_t idesc,
                                            uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n .reg .b64 b;\n mov.b64 b, {%2, %5};\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], b, %3, p;\n}\n" ::"r"(tmem_d),
      "r"(tmem_a), "r"(b_lo | kDescLo), "r"(idesc), "r"(accumulate), "r"(kDescHi)
      : "memory");
}
// one lane of the (converged) warp, the same one on every call
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n .reg .pred q;\n elect.sync _|q, 0xffffffff;\n selp.b32 %0, 1, 0, q;\n}\n" : "=r"(p));
  return p != 0;
}
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// TMEM transfers are aligned: all lanes of the warp at the instruction, so the two forms that follow code of some lanes
// alone (a ragged tile's stores, a barrier's arrival) converge first.
// 32 columns of this warp's lanes; complete on return (for the tensor core after fence_before and a barrier)
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
  __syncwarp();
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31};" ::"r"(r[0]),
      "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
      "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]),
      "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]),
      "r"(r[29]), "r"(r[30]), "r"(r[31]), "r"(taddr)
      : "memory");
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
  uint32_t r[32];
  __syncwarp();
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
}

// 16 columns, not yet complete (from a converged warp): tmem_ld_wait() follows the last of a batch, then tmem_loaded() on each
__device__ __forceinline__ void tmem_ld16_async(uint32_t taddr, float (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]), "=f"(v[8]),
        "=f"(v[9]), "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_loaded(float (&v)[16]) {  // no use of v moves ahead of the wait
#pragma unroll
  for (int j = 0; j < 16; ++j) asm volatile("" : "+f"(v[j]));
}

template <class TOUT> __device__ __forceinline__ TOUT cvt_out(float x);
template <> __device__ __forceinline__ float cvt_out<float>(float x) { return x; }
template <> __device__ __forceinline__ double cvt_out<double>(float x) { return (double)x; }
template <> __device__ __forceinline__ __half cvt_out<__half>(float x) { return __float2half_rn(x); }
template <> __device__ __forceinline__ __nv_bfloat16 cvt_out<__nv_bfloat16>(float x) { return __float2bfloat16_rn(x); }


typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline EncodeTiledFn get_encode() {
  static const EncodeTiledFn fn = [] {  // thread-safe one-time lookup
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      return (EncodeTiledFn)p;
    return (EncodeTiledFn) nullptr;
  }();
  return fn;
}

// 2D map over a K-contiguous operand: dims {K, rows}, row stride ld elements, box {64, box_rows}
inline bool make_map(CUtensorMap* map, ofrr_dtype t, const void* ptr, int64_t K, int64_t rows, int64_t ld,
                     int box_rows) {
  EncodeTiledFn enc = get_encode();
  if (!enc) return false;
  cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
  cuuint32_t box[2] = {(cuuint32_t)BK, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = enc(map, t == OFRR_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2,
                   const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

// 2D map over a K-contiguous byte operand (E4M3): dims {K, rows}, row stride ld bytes, box {128, box_rows}
inline bool make_map_u8(CUtensorMap* map, const void* ptr, int64_t K, int64_t rows, int64_t ld, int box_rows) {
  EncodeTiledFn enc = get_encode();
  if (!enc) return false;
  cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)ld};
  cuuint32_t box[2] = {(cuuint32_t)(2 * BK), (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(ptr), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

// kind::f16: F16 = 0, BF16 = 1; kind::f8f6f4: E4M3 = 0 (so the F16 encoding serves E4M3 operands)
inline uint32_t make_idesc(ofrr_dtype t, int BN) {
  const uint32_t fmt = (t == OFRR_BF16) ? 1u : 0u;
  uint32_t d = 0;
  d |= 1u << 4;                     // D format: F32
  d |= fmt << 7;                    // A format
  d |= fmt << 10;                   // B format
  d |= 0u << 15;                    // A K-major
  d |= 0u << 16;                    // B K-major
  d |= (uint32_t)(BN >> 3) << 17;   // N >> 3
  d |= (uint32_t)(BM >> 4) << 24;   // M >> 4
  return d;
}

}  // namespace tc
}  // namespace ofrr
