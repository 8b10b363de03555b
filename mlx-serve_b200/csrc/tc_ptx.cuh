// Shared by the tensor-core kernels (tcgen05 / TMA): mbarrier waits, bulk-tensor loads, operand descriptors, tensor-memory
// loads, the conversion of packed codes to bf16 weights, and the driver's tensor-map encoder.
#pragma once
#include <cuda.h>

#include <mutex>

#include "kernels.h"

namespace qb {

constexpr uint32_t kSpinLimit = 1u << 24;

// Bounded wait; returns false when the limit expired.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
  const uint32_t addr = smem_u32(bar);
  for (uint32_t it = 0; it < kSpinLimit; ++it) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(addr), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}
// The same for waits that are off the critical path (producers running ahead, the epilogue waiting for a
// whole tile): after a few polls the thread sleeps between polls, so that it does not take issue slots
// from the warps that convert weights.  Still bounded: 2^22 polls of at least 100 ns.
__device__ __forceinline__ bool mbar_wait_relaxed(uint64_t* bar, uint32_t parity) {
  const uint32_t addr = smem_u32(bar);
  for (uint32_t it = 0; it < (kSpinLimit >> 2); ++it) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(addr), "r"(parity)
        : "memory");
    if (done) return true;
    if (it >= 4) __nanosleep(100);
  }
  return false;
}
// Wait of the dequant warps: they run several stages ahead of the tensor core, so a poll that fails is followed
// by a short sleep -- sixteen warps polling in a tight loop take issue slots from the one thread that issues MMAs.
__device__ __forceinline__ bool mbar_wait_backoff(uint64_t* bar, uint32_t parity) {
  const uint32_t addr = smem_u32(bar);
  for (uint32_t it = 0; it < kSpinLimit; ++it) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(addr), "r"(parity)
        : "memory");
    if (done) return true;
    __nanosleep(40);
  }
  return false;
}
// The same with a number of polls of the caller's, each held by the hardware for kNap ns at most.
constexpr uint32_t kNap = 2000;
__device__ __forceinline__ bool wait_cta(uint64_t* bar, uint32_t parity, uint32_t polls) {
  const uint32_t addr = smem_u32(bar);
  for (uint32_t it = 0; it < polls; ++it) {
    uint32_t done;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(done) : "r"(addr), "r"(parity), "r"(kNap) : "memory");
    if (done) return true;
  }
  return false;
}
// One lane of a converged warp.  By elect.sync the compiler knows that it is one: behind it an MMA issues in 9 - 16 cycles, behind
// `lane == 0` in 73, commits and copies alike.
__device__ __forceinline__ bool elect_one() {
  uint32_t e;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(e));
  return e != 0;
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, uint64_t* bar, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
               ::"r"(dst), "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y)
               : "memory");
}
__device__ __forceinline__ uint32_t cluster_rank_tc() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ void cluster_sync_tc() {   // all threads of all CTAs of the cluster (hardware barrier)
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// K-major, SWIZZLE_128B operand descriptor: rows of 128 bytes, 8-row atoms 1024 bytes apart.
__device__ __forceinline__ uint64_t make_desc(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFF) >> 4);   // start address
  d |= (uint64_t)1 << 16;                    // leading byte offset (unused for swizzled K-major)
  d |= (uint64_t)(1024 >> 4) << 32;          // stride byte offset
  d |= (uint64_t)1 << 46;                    // descriptor version (Blackwell)
  d |= (uint64_t)2 << 61;                    // SWIZZLE_128B
  return d;
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,"
      "%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
}

// 32 codes (half of a k-block) of one weight row -> 32 bf16 values q*s+b (one rounding), written as
// chunks 4h..4h+3 of the 128-byte row `r` of a K-major SWIZZLE_128B tile (16-byte chunk c lands at
// chunk c ^ (r & 7)).
template <int BITS>
__device__ __forceinline__ void dequant_half(const uint32_t* codes, uint32_t sb2, uint32_t bb2, unsigned char* tile, int r,
                                             int h) {
  // sb2 / bb2: the group's scale / bias replicated in both bf16 lanes
  const __nv_bfloat162 s2 = *(const __nv_bfloat162*)&sb2, b2 = *(const __nv_bfloat162*)&bb2;
  unsigned char* row = tile + r * 128;
  const int xr = ((4 * h) ^ (r & 7)) << 4;   // chunk (4h + c) ^ (r & 7) = ((4h) ^ (r & 7)) ^ c for c < 4
  if constexpr (BITS == 4) {
    const __nv_bfloat162 c128 = __float2bfloat162_rn(128.f);
#pragma unroll
    for (int c = 0; c < 4; ++c) {  // one packed word = 8 values = one 16-byte chunk of bf16
      const uint32_t w = codes[c];
      // bytes (q1q0, q3q2, q5q4, q7q6) -> bytes q0,q1,q2,q3 and q4,q5,q6,q7 in order
      const uint32_t lo = __byte_perm(w, 0, 0x4140), hi = __byte_perm(w, 0, 0x4342);
      const uint32_t nl = (lo | (lo << 4)) & 0x0F0F0F0Fu, nh = (hi | (hi << 4)) & 0x0F0F0F0Fu;
      uint32_t o[4];
      // 0x43 in the high byte of a bf16 lane: 128 + q, exact
      o[0] = __byte_perm(nl, 0x43434343u, 0x5140);
      o[1] = __byte_perm(nl, 0x43434343u, 0x5342);
      o[2] = __byte_perm(nh, 0x43434343u, 0x5140);
      o[3] = __byte_perm(nh, 0x43434343u, 0x5342);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        __nv_bfloat162 v = *(__nv_bfloat162*)&o[j];
        v = __hsub2(v, c128);         // exact q
        v = __hfma2(v, s2, b2);       // q*s + b, rounded once
        o[j] = *(uint32_t*)&v;
      }
      *(uint4*)(row + (xr ^ (c << 4))) = make_uint4(o[0], o[1], o[2], o[3]);
    }
  } else {
#pragma unroll
    for (int c = 0; c < 4; ++c) {  // two packed words = 8 values
      uint32_t o[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t w = codes[2 * c + (j >> 1)], v = __byte_perm(w, 0, j & 1 ? 0x4342 : 0x4140);   // two codes in 16-bit halves
        const __nv_bfloat162 q = __hfma2(bf16_of_bytes(v), s2, b2);       // q*s + b, rounded once
        o[j] = *(uint32_t*)&q;
      }
      *(uint4*)(row + (xr ^ (c << 4))) = make_uint4(o[0], o[1], o[2], o[3]);
    }
  }
}

typedef CUresult (*EncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                             const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                             CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline EncodeFn get_encode() {
  static EncodeFn fn = nullptr;
  static bool tried = false;
  std::lock_guard<std::mutex> setup_lk(setup_mutex());
  if (!tried) {
    tried = true;
    void* sym = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = (EncodeFn)sym;
  }
  return fn;
}

// A matrix of `rows` rows of `cols` elements, `pitch` bytes apart, in boxes of br x bc; false where the driver declines it.
inline bool make_map(CUtensorMap* m, CUtensorMapDataType t, const void* base, int64_t cols, int64_t rows, int64_t pitch, int bc, int br,
                     CUtensorMapSwizzle swizzle = CU_TENSOR_MAP_SWIZZLE_128B) {
  const EncodeFn enc = get_encode();
  const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)pitch};
  const cuuint32_t box[2] = {(cuuint32_t)bc, (cuuint32_t)br}, es[2] = {1, 1};
  return enc && enc(m, t, 2, (void*)base, dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace qb
