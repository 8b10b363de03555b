// Shared device/host helpers for libqb200 (sm_100a only).
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/qb200.h"

namespace qb {

constexpr int kMaxLead = QB200_MAX_DIMS - 1;  // leading (row) dims of a tensor

// Maps a linear row index (row-major over `nd` leading dims) to an element
// offset using explicit strides.  Cache views are strided slices of capacity
// buffers (mlx-serve src/transformer.zig:3472-3495), so every kernel that
// walks rows of a caller tensor goes through one of these.
struct RowMap {
  int nd;
  int64_t shape[kMaxLead];
  int64_t stride[kMaxLead];
  int contiguous;      // rows are `row_pitch` elements apart, no gaps
  int64_t row_pitch;
  __host__ __device__ inline int64_t offset(int64_t row) const {
    if (contiguous) return row * row_pitch;
    int64_t off = 0;
    for (int d = nd - 1; d >= 0; --d) {
      const int64_t q = row / shape[d];
      off += (row - q * shape[d]) * stride[d];
      row = q;
    }
    return off;
  }
};

// Broadcast batch addressing for matmul operands: batch index -> element offset.
struct BatchMap {
  int nd;
  int64_t shape[kMaxLead];    // broadcast batch shape
  int64_t stride[kMaxLead];   // 0 where the operand is broadcast
  __host__ __device__ inline int64_t offset(int64_t bidx) const {
    int64_t off = 0;
    for (int d = nd - 1; d >= 0; --d) {
      const int64_t q = bidx / shape[d];
      off += (bidx - q * shape[d]) * stride[d];
      bidx = q;
    }
    return off;
  }
};

__device__ __forceinline__ float bf16_bits_to_f32(uint16_t h) { return __uint_as_float(((uint32_t)h) << 16); }
__device__ __forceinline__ float bf16lo(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float bf16hi(uint32_t v) { return __uint_as_float(v & 0xFFFF0000u); }
__device__ __forceinline__ uint16_t f32_to_bf16_bits(float f) {
  return __bfloat16_as_ushort(__float2bfloat16_rn(f));
}
__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
  return (uint32_t)f32_to_bf16_bits(lo) | ((uint32_t)f32_to_bf16_bits(hi) << 16);
}

// two fp32 -> packed bf16 (round to nearest even), `lo` in the low half: one conversion instruction
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
  return *(const uint32_t*)&h;
}

// sigmoid of a bf16 value, rounded to bf16: the two-sided form of MLX's Sigmoid as the reference quotes it
// (src/transformer.zig:17566-17570).  The approximate exponential and reciprocal give the same bf16 as fp32 libm for every
// one of the 65536 patterns with |x| <= 80 (the elementwise tests go through all of them); beyond, where the result is
// subnormal, the exact functions do.
__device__ __forceinline__ float sigmoid_bf16(float x) {
  const float ax = fabsf(x);
  float e, r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(ax * 1.4426950408889634f));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(1.f + e));
  if (ax > 80.f) r = 1.f / (1.f + expf(ax));
  return bf16_bits_to_f32(f32_to_bf16_bits(x < 0.f ? r : 1.f - r));
}

template <typename T> struct IO;
template <> struct IO<float> {
  __device__ static __forceinline__ float load(const void* p, int64_t i) { return ((const float*)p)[i]; }
  __device__ static __forceinline__ void store(void* p, int64_t i, float v) { ((float*)p)[i] = v; }
};
template <> struct IO<__nv_bfloat16> {
  __device__ static __forceinline__ float load(const void* p, int64_t i) {
    return bf16_bits_to_f32(((const uint16_t*)p)[i]);
  }
  __device__ static __forceinline__ void store(void* p, int64_t i, float v) {
    ((uint16_t*)p)[i] = f32_to_bf16_bits(v);
  }
};
template <> struct IO<__half> {
  __device__ static __forceinline__ float load(const void* p, int64_t i) { return __half2float(((const __half*)p)[i]); }
  __device__ static __forceinline__ void store(void* p, int64_t i, float v) { ((__half*)p)[i] = __float2half_rn(v); }
};

// Streaming 64/128-bit loads of packed weights: read-only path, do not keep in L1.
__device__ __forceinline__ uint2 ldg_stream_u2(const void* p) {
  uint2 v;
  asm volatile("ld.global.nc.L1::no_allocate.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
  return v;
}
__device__ __forceinline__ uint4 ldg_stream_u4(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p));
  return v;
}
__device__ __forceinline__ uint32_t ldg_stream_u32(const void* p) {
  uint32_t v;
  asm volatile("ld.global.nc.L1::no_allocate.u32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}

// D(16x8,f32) += A(16x16,bf16,row) * B(16x8,bf16,col)
__device__ __forceinline__ void mma_bf16_16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// D(16x8,f32) += A(16x16,f16,row) * B(16x8,f16,col)
__device__ __forceinline__ void mma_f16_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm(  // not volatile: the scheduler may interleave independent accumulation chains

      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// D(16x8,f32) += A(16x8,bf16) * B(8x8,bf16)
__device__ __forceinline__ void mma_bf16_1688(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t b) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(b));
}
__device__ __forceinline__ float pow2i(int e) { return __uint_as_float((uint32_t)(e + 127) << 23); }   // 2^e, e in [-126, 127]
// two fp32 -> packed fp16 (round to nearest even), `lo` in the low half
__device__ __forceinline__ uint32_t pack_f16x2(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}

// The same as mma_bf16_16816 with a zero C operand.
__device__ __forceinline__ void mma_bf16_16816_z(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}

// (a & b) | c in one LOP3
__device__ __forceinline__ uint32_t lop3_and_or(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t r;
  asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
  return r;
}

// The bytes 0 and 2 of a word as exact bf16 integers 0..255: 128 + the low seven bits, minus 128 where the top bit is clear
// (0x80 * 0x186 = 0xC300 = -128).
__device__ __forceinline__ __nv_bfloat162 bf16_of_bytes(uint32_t v) {
  const uint32_t lo = lop3_and_or(v, 0x007F007Fu, 0x43004300u), hi = ((v & 0x00800080u) ^ 0x00800080u) * 0x186u;
  return __hadd2(*(const __nv_bfloat162*)&lo, *(const __nv_bfloat162*)&hi);
}

// ---- mbarriers of this CTA, by their shared-memory address or by pointer ----
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) { mbar_init(smem_u32(bar), count); }
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) { mbar_arrive(smem_u32(bar)); }
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

}  // namespace qb
