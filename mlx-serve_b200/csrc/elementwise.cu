// dequantize / quantize kernels (bit-exact against the CPU oracle).
//
// dequantize mirrors mlx_dequantize as used by kv_quant.dequantizeAffine
// (mlx-serve src/kv_quant.zig:407-430): w = q*scale + bias with a rounded fp32
// product and a rounded fp32 add (no FMA contraction), then one cast.
// quantize mirrors mlx_quantize as used by kv_quant.quantizeAffine
// (src/kv_quant.zig:126-162); the scale/bias rule is the one restated in
// tests/dsv4_imatrix.py:169-183 and the codes follow :264.
#include "kernels.h"

namespace qb {

namespace {

template <typename T> struct DT;
template <> struct DT<float> { static constexpr int v = QB200_FLOAT32; };
template <> struct DT<__nv_bfloat16> { static constexpr int v = QB200_BFLOAT16; };
template <> struct DT<__half> { static constexpr int v = QB200_FLOAT16; };

template <int BITS, typename ST, typename OT>
__global__ void __launch_bounds__(256) dequant_kernel(DequantArgs a, int64_t words_per_row, int64_t total_words) {
  constexpr int VPW = 32 / BITS;
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= total_words) return;
  const int64_t row = idx / words_per_row;
  const int64_t wi = idx - row * words_per_row;
  const uint32_t word = a.w[a.wmap.offset(row) + wi];
  const int64_t g = (wi * VPW) / a.gs;
  const int64_t sboff = a.sbmap.offset(row) + g;
  const float sc = IO<ST>::load(a.s, sboff);
  const float bi = IO<ST>::load(a.b, sboff);
  const int64_t obase = a.omap.offset(row) + wi * VPW;
  float v[VPW];
#pragma unroll
  for (int k = 0; k < VPW; ++k) {
    const float q = (float)((word >> (k * BITS)) & ((1u << BITS) - 1u));
    v[k] = __fadd_rn(__fmul_rn(q, sc), bi);
  }
  if constexpr (sizeof(OT) == 2 && VPW % 2 == 0) {
    // packed 16-bit stores when the destination is suitably aligned
    OT* op = (OT*)a.out + obase;
    if ((((uintptr_t)op) & (VPW * 2 - 1)) == 0) {
      uint32_t pk[VPW / 2];
#pragma unroll
      for (int k = 0; k < VPW / 2; ++k) {
        OT lo, hi;
        if constexpr (DT<OT>::v == QB200_BFLOAT16) { lo = __float2bfloat16_rn(v[2 * k]); hi = __float2bfloat16_rn(v[2 * k + 1]); }
        else { lo = __float2half_rn(v[2 * k]); hi = __float2half_rn(v[2 * k + 1]); }
        pk[k] = (uint32_t)(*(uint16_t*)&lo) | ((uint32_t)(*(uint16_t*)&hi) << 16);
      }
      if constexpr (VPW == 8) *(uint4*)op = make_uint4(pk[0], pk[1], pk[2], pk[3]);
      else if constexpr (VPW == 4) *(uint2*)op = make_uint2(pk[0], pk[1]);
      else {
#pragma unroll
        for (int k = 0; k < VPW / 2; ++k) ((uint32_t*)op)[k] = pk[k];
      }
      return;
    }
  }
#pragma unroll
  for (int k = 0; k < VPW; ++k) IO<OT>::store(a.out, obase + k, v[k]);
}

template <int BITS, typename ST>
cudaError_t dequant_dispatch_out(const DequantArgs& a, cudaStream_t st) {
  const int64_t wpr = a.d * BITS / 32;
  const int64_t total = a.rows * wpr;
  if (total == 0) return cudaSuccess;
  const unsigned blocks = (unsigned)((total + 255) / 256);
  switch (a.out_dtype) {
    case QB200_BFLOAT16: dequant_kernel<BITS, ST, __nv_bfloat16><<<blocks, 256, 0, st>>>(a, wpr, total); break;
    case QB200_FLOAT32: dequant_kernel<BITS, ST, float><<<blocks, 256, 0, st>>>(a, wpr, total); break;
    case QB200_FLOAT16: dequant_kernel<BITS, ST, __half><<<blocks, 256, 0, st>>>(a, wpr, total); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

template <int BITS>
cudaError_t dequant_dispatch_sb(const DequantArgs& a, cudaStream_t st) {
  switch (a.sb_dtype) {
    case QB200_BFLOAT16: return dequant_dispatch_out<BITS, __nv_bfloat16>(a, st);
    case QB200_FLOAT32: return dequant_dispatch_out<BITS, float>(a, st);
    case QB200_FLOAT16: return dequant_dispatch_out<BITS, __half>(a, st);
    default: return cudaErrorInvalidValue;
  }
}

// One thread per packed output word; the gs/VPW threads of a group are
// consecutive lanes of one warp and share min/max through shuffles.
template <int BITS, typename XT, typename ST>
__global__ void __launch_bounds__(256) quant_kernel(QuantArgs a, int64_t words_per_row, int64_t total_words) {
  constexpr int VPW = 32 / BITS;
  int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool live = idx < total_words;
  if (!live) idx = total_words - 1;  // keep the warp converged for the shuffles
  const int64_t row = idx / words_per_row;
  const int64_t wi = idx - row * words_per_row;
  const int64_t xbase = a.xmap.offset(row) + wi * VPW;
  float v[VPW];
#pragma unroll
  for (int k = 0; k < VPW; ++k) v[k] = IO<XT>::load(a.x, xbase + k);
  float xmin = v[0], xmax = v[0];
#pragma unroll
  for (int k = 1; k < VPW; ++k) { xmin = fminf(xmin, v[k]); xmax = fmaxf(xmax, v[k]); }
  const int tpg = a.gs / VPW;  // threads per group: power of two, <= 32
  for (int off = tpg >> 1; off > 0; off >>= 1) {
    xmin = fminf(xmin, __shfl_xor_sync(0xffffffffu, xmin, off));
    xmax = fmaxf(xmax, __shfl_xor_sync(0xffffffffu, xmax, off));
  }
  const float n_bins = (float)((1 << BITS) - 1);
  const bool mask = fabsf(xmin) > fabsf(xmax);
  float scale = fmaxf(__fdiv_rn(__fsub_rn(xmax, xmin), n_bins), 1e-7f);
  scale = mask ? scale : -scale;
  const float edge = mask ? xmin : xmax;
  const float q0 = rintf(__fdiv_rn(edge, scale));
  float bias = 0.0f;
  if (q0 != 0.0f) { scale = __fdiv_rn(edge, q0); bias = edge; }
  uint32_t word = 0;
#pragma unroll
  for (int k = 0; k < VPW; ++k) {
    float c = rintf(__fdiv_rn(__fsub_rn(v[k], bias), scale));
    c = fminf(fmaxf(c, 0.0f), n_bins);
    word |= ((uint32_t)c) << (k * BITS);
  }
  if (!live) return;
  a.q[a.qmap.offset(row) + wi] = word;
  if ((wi % tpg) == 0) {
    const int64_t sboff = a.sbmap.offset(row) + (wi * VPW) / a.gs;
    IO<ST>::store(a.s, sboff, scale);
    IO<ST>::store(a.b, sboff, bias);
  }
}

template <int BITS, typename XT>
cudaError_t quant_dispatch_sb(const QuantArgs& a, cudaStream_t st) {
  const int64_t wpr = a.d * BITS / 32;
  const int64_t total = a.rows * wpr;
  if (total == 0) return cudaSuccess;
  const unsigned blocks = (unsigned)((total + 255) / 256);
  switch (a.sb_dtype) {
    case QB200_BFLOAT16: quant_kernel<BITS, XT, __nv_bfloat16><<<blocks, 256, 0, st>>>(a, wpr, total); break;
    case QB200_FLOAT32: quant_kernel<BITS, XT, float><<<blocks, 256, 0, st>>>(a, wpr, total); break;
    case QB200_FLOAT16: quant_kernel<BITS, XT, __half><<<blocks, 256, 0, st>>>(a, wpr, total); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

template <int BITS>
cudaError_t quant_dispatch_x(const QuantArgs& a, cudaStream_t st) {
  switch (a.x_dtype) {
    case QB200_BFLOAT16: return quant_dispatch_sb<BITS, __nv_bfloat16>(a, st);
    case QB200_FLOAT32: return quant_dispatch_sb<BITS, float>(a, st);
    case QB200_FLOAT16: return quant_dispatch_sb<BITS, __half>(a, st);
    default: return cudaErrorInvalidValue;
  }
}

// ---- the same two operators for bf16 tensors, 4 or 8 bits, rows of 16-byte aligned values ----
// HBM-bound: 16 values per thread, 16-byte accesses on the dense side, the row's offsets from a (block, row) pair instead of
// 64-bit divisions per element.  K and V of 2 x 8 x 4096 tokens at head dim 128, 8 bits, appended and read back as bf16 (87 MB):
// 168 us with the element-wise kernels above, which stay for other dtypes, 2 bits and unaligned rows.
constexpr int kRowVals = 16;    // values per thread: the group's parameters (four divisions) are worked out once per 16

// Rows as z x y x inner; each tensor's element strides along the three.
struct RowAxis { int64_t z, y, inner; };
struct RowGrid {
  int nz, ny, inner;            // blockIdx.z, blockIdx.y, rows per (z, y)
  int per_row, shift;           // threads per row (d / kRowVals), its log2 or -1
};
__device__ __forceinline__ int64_t row_base(const RowAxis& m, int row) { return blockIdx.z * m.z + blockIdx.y * m.y + row * m.inner; }
__device__ __forceinline__ int row_of(const RowGrid& rg, int i) { return rg.shift >= 0 ? i >> rg.shift : (int)((uint32_t)i / (uint32_t)rg.per_row); }

// rint(x / s) clamped to [0, bins], exactly as the division rounds: away from the ties the product with 1 / s decides, near
// them (within 2^-10, far more than its error for quotients up to 256) and where anything is not finite the division does.
__device__ __forceinline__ uint32_t code_of(float x, float bias, float s, float rs, float bins) {
  const float n = __fsub_rn(x, bias);
  const float t = fmaf(n, rs, 12582912.f);          // 1.5 * 2^23 + rint(n / s): the low bits are the integer
  const float r = fmaf(n, rs, 12582912.f - t);      // what the rounding left
  float c = t - 12582912.f;
  if (!(fabsf(r) < 0.5f - 9.765625e-4f)) c = rintf(__fdiv_rn(n, s));
  return (uint32_t)fminf(fmaxf(c, 0.0f), bins);
}

template <int BITS>
__global__ void __launch_bounds__(256) quant_rows_kernel(const uint16_t* x, uint32_t* qo, uint16_t* so, uint16_t* bo, RowAxis ax, RowAxis aq, RowAxis as,
                                                         RowGrid rg, int gs) {
  const int i = blockIdx.x * 256 + threadIdx.x;
  const bool live = i < rg.inner * rg.per_row;
  const int row = live ? row_of(rg, i) : 0, c = live ? i - row * rg.per_row : 0;
  const uint16_t* xp = x + row_base(ax, row) + c * kRowVals;
  float v[kRowVals];
#pragma unroll
  for (int k = 0; k < kRowVals / 8; ++k) {
    const uint4 raw = ((const uint4*)xp)[k];
    const uint32_t q[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) { v[8 * k + 2 * j] = bf16lo(q[j]); v[8 * k + 2 * j + 1] = bf16hi(q[j]); }
  }
  float xmin = v[0], xmax = v[0];
#pragma unroll
  for (int k = 1; k < kRowVals; ++k) { xmin = fminf(xmin, v[k]); xmax = fmaxf(xmax, v[k]); }
  const int tpg = gs / kRowVals;   // neighbouring lanes share a group: 2, 4 or 8
  for (int off = tpg >> 1; off > 0; off >>= 1) {
    xmin = fminf(xmin, __shfl_xor_sync(0xffffffffu, xmin, off));
    xmax = fmaxf(xmax, __shfl_xor_sync(0xffffffffu, xmax, off));
  }
  const float n_bins = (float)((1 << BITS) - 1);
  const bool mask = fabsf(xmin) > fabsf(xmax);
  float scale = fmaxf(__fdiv_rn(__fsub_rn(xmax, xmin), n_bins), 1e-7f);
  scale = mask ? scale : -scale;
  const float edge = mask ? xmin : xmax;
  const float q0 = rintf(__fdiv_rn(edge, scale));
  float bias = 0.0f;
  if (q0 != 0.0f) { scale = __fdiv_rn(edge, q0); bias = edge; }
  const float rs = __fdiv_rn(1.0f, scale);
  uint32_t w[BITS / 2] = {};
#pragma unroll
  for (int k = 0; k < kRowVals; ++k) w[k * BITS / 32] |= code_of(v[k], bias, scale, rs, n_bins) << (k * BITS % 32);
  if (!live) return;
  uint32_t* qp = qo + row_base(aq, row) + c * (BITS / 2);
  if constexpr (BITS == 4) *(uint2*)qp = make_uint2(w[0], w[1]); else *(uint4*)qp = make_uint4(w[0], w[1], w[BITS / 2 - 2], w[BITS / 2 - 1]);
  if ((c & (tpg - 1)) == 0) {
    const int64_t sb = row_base(as, row) + c / tpg;
    so[sb] = f32_to_bf16_bits(scale);
    bo[sb] = f32_to_bf16_bits(bias);
  }
}

template <int BITS>
__global__ void __launch_bounds__(256) dequant_rows_kernel(const uint32_t* wq, const uint16_t* s, const uint16_t* b, uint16_t* out, RowAxis aw, RowAxis as,
                                                           RowAxis ao, RowGrid rg, int gs) {
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i >= rg.inner * rg.per_row) return;
  const int row = row_of(rg, i), c = i - row * rg.per_row;
  const uint32_t* wp = wq + row_base(aw, row) + c * (BITS / 2);
  uint32_t w[BITS / 2];
  if constexpr (BITS == 4) { const uint2 q = *(const uint2*)wp; w[0] = q.x; w[1] = q.y; }
  else { const uint4 q = *(const uint4*)wp; w[0] = q.x; w[1] = q.y; w[BITS / 2 - 2] = q.z; w[BITS / 2 - 1] = q.w; }
  const int64_t sb = row_base(as, row) + c / (gs / kRowVals);
  const float sc = bf16_bits_to_f32(s[sb]), bi = bf16_bits_to_f32(b[sb]);
  float v[kRowVals];
#pragma unroll
  for (int k = 0; k < kRowVals; ++k) {
    // the code as a float: 2^23 + c, minus 2^23
    const float q = __uint_as_float(((w[k * BITS / 32] >> (k * BITS % 32)) & ((1u << BITS) - 1u)) | 0x4B000000u) - 8388608.f;
    v[k] = __fadd_rn(__fmul_rn(q, sc), bi);
  }
  uint16_t* op = out + row_base(ao, row) + c * kRowVals;
#pragma unroll
  for (int k = 0; k < kRowVals; k += 8)
    *(uint4*)(op + k) = make_uint4(pack2(v[k], v[k + 1]), pack2(v[k + 2], v[k + 3]), pack2(v[k + 4], v[k + 5]), pack2(v[k + 6], v[k + 7]));
}

// Every row offset of `m` is a multiple of `unit` elements.
bool rows_aligned(const RowMap& m, int64_t unit) {
  for (int d = 0; d < m.nd; ++d)
    if (m.shape[d] != 1 && m.stride[d] % unit != 0) return false;
  return true;
}
// Splits the rows into z x y x inner with one stride each per tensor; false where that takes more axes or the grid would not
// hold them.
bool row_grid(const RowMap* const (&maps)[3], int64_t rows, int64_t d, RowGrid* rg, RowAxis (&ax)[3]) {
  const RowMap& m0 = *maps[0];
  const bool flat = maps[0]->contiguous && maps[1]->contiguous && maps[2]->contiguous;
  if (!flat && m0.nd > 3) return false;
  const int64_t ext[3] = {!flat && m0.nd > 2 ? m0.shape[m0.nd - 3] : 1, !flat && m0.nd > 1 ? m0.shape[m0.nd - 2] : 1, flat ? rows : m0.shape[m0.nd - 1]};
  for (int i = 0; i < 3; ++i) {
    const RowMap& m = *maps[i];
    ax[i].z = !flat && m.nd > 2 ? m.stride[m.nd - 3] : 0;
    ax[i].y = !flat && m.nd > 1 ? m.stride[m.nd - 2] : 0;
    ax[i].inner = flat ? m.row_pitch : m.stride[m.nd - 1];
  }
  if (d % kRowVals != 0 || d / kRowVals > (1 << 24) || ext[2] * (d / kRowVals) > (int64_t)1 << 30 || ext[0] > 65535 || ext[1] > 65535) return false;
  rg->nz = (int)ext[0]; rg->ny = (int)ext[1]; rg->inner = (int)ext[2];
  rg->per_row = (int)(d / kRowVals);
  rg->shift = -1;
  for (int k = 0; k < 24; ++k)
    if (rg->per_row == 1 << k) rg->shift = k;
  return true;
}
dim3 row_blocks(const RowGrid& rg) { return dim3((unsigned)(((int64_t)rg.inner * rg.per_row + 255) / 256), (unsigned)rg.ny, (unsigned)rg.nz); }

bool quant_rows(const QuantArgs& a, cudaStream_t st, cudaError_t* e) {
  if ((a.bits != 4 && a.bits != 8) || a.x_dtype != QB200_BFLOAT16 || a.sb_dtype != QB200_BFLOAT16) return false;
  if (((uintptr_t)a.x & 15) || !rows_aligned(a.xmap, 8) || ((uintptr_t)a.q & (2 * a.bits - 1)) || !rows_aligned(a.qmap, a.bits / 2)) return false;
  const RowMap* const maps[3] = {&a.xmap, &a.qmap, &a.sbmap};
  RowGrid rg;
  RowAxis ax[3];
  if (!row_grid(maps, a.rows, a.d, &rg, ax)) return false;
  auto kern = a.bits == 4 ? quant_rows_kernel<4> : quant_rows_kernel<8>;
  kern<<<row_blocks(rg), 256, 0, st>>>((const uint16_t*)a.x, a.q, (uint16_t*)a.s, (uint16_t*)a.b, ax[0], ax[1], ax[2], rg, a.gs);
  *e = cudaGetLastError();
  return true;
}
bool dequant_rows(const DequantArgs& a, cudaStream_t st, cudaError_t* e) {
  if ((a.bits != 4 && a.bits != 8) || a.out_dtype != QB200_BFLOAT16 || a.sb_dtype != QB200_BFLOAT16) return false;
  if (((uintptr_t)a.out & 15) || !rows_aligned(a.omap, 8) || ((uintptr_t)a.w & (2 * a.bits - 1)) || !rows_aligned(a.wmap, a.bits / 2)) return false;
  const RowMap* const maps[3] = {&a.wmap, &a.sbmap, &a.omap};
  RowGrid rg;
  RowAxis ax[3];
  if (!row_grid(maps, a.rows, a.d, &rg, ax)) return false;
  auto kern = a.bits == 4 ? dequant_rows_kernel<4> : dequant_rows_kernel<8>;
  kern<<<row_blocks(rg), 256, 0, st>>>(a.w, (const uint16_t*)a.s, (const uint16_t*)a.b, (uint16_t*)a.out, ax[0], ax[1], ax[2], rg, a.gs);
  *e = cudaGetLastError();
  return true;
}

// One thread per 8 consecutive h of one token: the k rows are read 16 bytes at a time.  bf16: every product is
// rounded to bf16 (the reference multiplies in the activation dtype, src/transformer.zig:15127-15140) and the sum
// over k is an ascending accumulate in bf16, rounded after every add, which is how MLX reduces a bf16 row and what
// the reference's fused down+reduce kernel replicates (src/transformer.zig:20566-20571).
template <bool F32>
__global__ void __launch_bounds__(256) moe_sum_kernel(MoeSumArgs a) {
  const int64_t per_tok = a.H / 8;
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.T * per_tok) return;
  const int64_t t = i / per_tok, h0 = (i - t * per_tok) * 8;
  float acc[8];
  __nv_bfloat162 accp[4];   // bf16: packed, the packed operations round exactly where the scalar form would
#pragma unroll
  for (int j = 0; j < 8; ++j) acc[j] = 0.f;
#pragma unroll
  for (int j = 0; j < 4; ++j) accp[j] = __float2bfloat162_rn(0.f);
  // top-k entries in batches of 8: first every index and score, then every row (independent loads in flight
  // together), then the products in ascending j
  for (int64_t j0 = 0; j0 < a.topk; j0 += 8) {
    int64_t row[8];
    float sc[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int64_t e = t * a.topk + j0 + q;
      row[q] = -1;
      sc[q] = 0.f;
      if (j0 + q < a.topk) {
        row[q] = a.inv ? (a.inv_i64 ? ((const long long*)a.inv)[e] : (long long)((const int*)a.inv)[e]) : e;
        sc[q] = F32 ? ((const float*)a.scores)[e] : __uint_as_float((uint32_t)((const uint16_t*)a.scores)[e] << 16);
        if (row[q] >= a.R) row[q] = -1;   // out-of-range (and negative) entries contribute nothing
      }
    }
    uint4 v0[8], v1[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      v0[q] = v1[q] = make_uint4(0u, 0u, 0u, 0u);
      if (row[q] >= 0) {
        if (F32) {
          v0[q] = *(const uint4*)((const float*)a.y + row[q] * a.H + h0);
          v1[q] = *(const uint4*)((const float*)a.y + row[q] * a.H + h0 + 4);
        } else {
          v0[q] = *(const uint4*)((const uint16_t*)a.y + row[q] * a.H + h0);
        }
      }
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      if (row[q] < 0) continue;
      if (F32) {
        const uint32_t w[8] = {v0[q].x, v0[q].y, v0[q].z, v0[q].w, v1[q].x, v1[q].y, v1[q].z, v1[q].w};
#pragma unroll
        for (int c = 0; c < 8; ++c) acc[c] += __uint_as_float(w[c]) * sc[q];
      } else {
        const uint32_t w[4] = {v0[q].x, v0[q].y, v0[q].z, v0[q].w};
        const __nv_bfloat162 s2 = __float2bfloat162_rn(sc[q]);
#pragma unroll
        for (int c = 0; c < 4; ++c)     // product rounded to bf16, then a bf16 accumulate (rounded after every add)
          accp[c] = __hadd2_rn(accp[c], __hmul2_rn(*(const __nv_bfloat162*)&w[c], s2));
      }
    }
  }
  if (F32) {
    float* o = (float*)a.out + t * a.H + h0;
    *(float4*)o = make_float4(acc[0], acc[1], acc[2], acc[3]);
    *(float4*)(o + 4) = make_float4(acc[4], acc[5], acc[6], acc[7]);
  } else {
    const uint4 o = *(const uint4*)accp;
    *(uint4*)((uint16_t*)a.out + t * a.H + h0) = o;
  }
}

// One warp per row of logits (E <= 1024: up to 32 values per lane, column e in lane e % 32).  The k indices are
// those of the largest logits, larger first, equal logits by lower index (the reference takes them from
// mlx_argpartition, which leaves their order open; everything downstream is indexed alike, src/transformer.zig:17022-17063).
// softmax in fp32 (precise), rounded to the logits' dtype as the reference's array is, then the k entries divided
// by their sum (accumulated in that dtype, larger-first order), each step rounded to that dtype -- the order and the
// accumulation are those of the reference's one-kernel router (src/transformer.zig:17485-17500, :17530-17534).
// kPer: values per lane.  A selection round is two warp reductions (the largest key, the lowest index that has it) instead of
// five rounds of two shuffles, and the probabilities of the k selected are worked out side by side after the last one:
// 4096 rows of 128 took 26 us with 32 values per lane whatever E was.
template <bool F32, int kPer>
__global__ void __launch_bounds__(128) moe_route_kernel(MoeRouteArgs a) {
  const int lane = threadIdx.x & 31;
  const int64_t row = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= a.T) return;
  float v[kPer];
  float mx = -INFINITY;
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    const int e = i * 32 + lane;
    v[i] = -INFINITY;
    if (e < a.E) {
      v[i] = F32 ? ((const float*)a.logits)[row * a.E + e]
                 : __uint_as_float((uint32_t)((const uint16_t*)a.logits)[row * a.E + e] << 16);
      mx = fmaxf(mx, v[i]);
    }
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, d));
  float sum = 0.f;
#pragma unroll
  for (int i = 0; i < kPer; ++i)
    if (i * 32 + lane < a.E) sum += expf(v[i] - mx);
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, d);
  auto round_dt = [](float x) { return F32 ? x : __uint_as_float((uint32_t)f32_to_bf16_bits(x) << 16); };
  // keys that order like the values (-0 like 0); 0 = not selectable (behind E, a NaN, already selected)
  uint32_t key[kPer];
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    const uint32_t u = __float_as_uint(v[i] + 0.f);
    key[i] = (i * 32 + lane < a.E && v[i] == v[i]) ? ((u >> 31) ? ~u : (u | 0x80000000u)) : 0u;
  }
  uint32_t my_key = 0;             // lane j keeps the j-th selected
  int my_idx = 0;
  for (int j = 0; j < a.topk; ++j) {
    uint32_t bk = 0;
    int bi = 0x7fffffff;
#pragma unroll
    for (int i = 0; i < kPer; ++i)
      if (key[i] > bk) { bk = key[i]; bi = i * 32 + lane; }
    const uint32_t m = __reduce_max_sync(0xffffffffu, bk);
    const int e = m ? __reduce_min_sync(0xffffffffu, bk == m ? bi : 0x7fffffff) : 0x7fffffff;
    if (m && (e & 31) == lane) {
#pragma unroll
      for (int i = 0; i < kPer; ++i)
        if (i == (e >> 5)) key[i] = 0u;
    }
    if (lane == j) { my_key = m; my_idx = m ? e : 0; }
  }
  const float bv = __uint_as_float((my_key >> 31) ? (my_key & 0x7FFFFFFFu) : ~my_key);
  const float topw = my_key ? round_dt(expf(bv - mx) / sum) : 0.f;
  float wsum = 0.f;
  for (int j = 0; j < a.topk; ++j)   // ascending accumulate in the logits' dtype, rounded after every add (src/transformer.zig:17530-17534)
    wsum = round_dt(wsum + __shfl_sync(0xffffffffu, topw, j));
  if (lane < a.topk) {
    a.inds[row * a.topk + lane] = my_idx;
    const float ns = round_dt(topw / wsum);
    if (F32) ((float*)a.scores)[row * a.topk + lane] = ns;
    else ((uint16_t*)a.scores)[row * a.topk + lane] = f32_to_bf16_bits(ns);
  }
}

template <bool F32>
cudaError_t route_dispatch(const MoeRouteArgs& a, cudaStream_t st) {
  const int warps = a.T >= 4 * sm_count() ? 4 : 1;   // few rows: a CTA each, so that every one has an SM to itself
  const unsigned blocks = (unsigned)((a.T + warps - 1) / warps);
  if (a.E <= 128) moe_route_kernel<F32, 4><<<blocks, warps * 32, 0, st>>>(a);
  else if (a.E <= 256) moe_route_kernel<F32, 8><<<blocks, warps * 32, 0, st>>>(a);
  else moe_route_kernel<F32, 32><<<blocks, warps * 32, 0, st>>>(a);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_moe_route(const MoeRouteArgs& a, cudaStream_t st) {
  if (a.T <= 0) return cudaSuccess;
  return a.dtype == QB200_FLOAT32 ? route_dispatch<true>(a, st) : route_dispatch<false>(a, st);
}

cudaError_t launch_moe_weighted_sum(const MoeSumArgs& a, cudaStream_t st) {
  const int64_t n = a.T * (a.H / 8);
  if (n <= 0) return cudaSuccess;
  const unsigned blocks = (unsigned)((n + 255) / 256);
  if (a.dtype == QB200_FLOAT32) moe_sum_kernel<true><<<blocks, 256, 0, st>>>(a);
  else moe_sum_kernel<false><<<blocks, 256, 0, st>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_dequantize(const DequantArgs& a, cudaStream_t st) {
  cudaError_t e;
  if (dequant_rows(a, st, &e)) return e;
  switch (a.bits) {
    case 2: return dequant_dispatch_sb<2>(a, st);
    case 4: return dequant_dispatch_sb<4>(a, st);
    case 8: return dequant_dispatch_sb<8>(a, st);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_quantize(const QuantArgs& a, cudaStream_t st) {
  cudaError_t e;
  if (quant_rows(a, st, &e)) return e;
  switch (a.bits) {
    case 2: return quant_dispatch_x<2>(a, st);
    case 4: return quant_dispatch_x<4>(a, st);
    case 8: return quant_dispatch_x<8>(a, st);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace qb
