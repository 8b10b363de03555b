// Tiled quantized matmul with the weight term in fp32, for widths the tcgen05 kernel does not take: y[M, N] = x[M, K] . What^T,
// bf16 activations, 4- or 8-bit affine codes, group size 32 / 64 / 128, K any multiple of the group size, from 5 tokens on (which of them: the rule in api.cu);
// and the same over rows sorted by expert (gather_qmm).
//
// Replaces mlx_quantized_matmul / mlx_gather_qmm (transpose = true; mlx-serve src/transformer.zig:20894-20983, :20763-20784) at
// such shapes, which ran on the CUDA cores (about 4 TFLOP/s; dense ones then in 32-token passes of the streaming kernel).
//
// Bound: at hundreds of tokens the rate of the warp-level MMA (about 580 TFLOP/s of m16n8k16 on this part); at tens of tokens the
// dependent chain of a stage and its barrier (27 x 12000 x 4416: tensor pipe 27 % active, issue 0.40 per scheduler).  The weight term must not be rounded here,
// so the MMA multiplies the codes themselves, and every group's sums are scaled in fp32 (one FMA per output against four MMAs,
// which take four times the issue slots' time).  tcgen05 would need an accumulator per group in tensor memory and the same
// FMAs after reading it back; it serves the rounded-weight shapes instead.
//  * CTA: 8 warps on a tile of TM tokens x 32 WN weight rows, K in stages of 64 through a ring of cp.async copies of x and W as
//    they are; one barrier per stage.
//  * Codes become bf16 integers in registers: 4 bits 128 + c (a shift and a LOP3 per two codes), 8 bits exactly c.  The pairs cut
//    out of a packed word are not neighbours in k; the activations' pairs are permuted alike (a byte permutation each).
//  * y = sum_g s_g (d_g - 128 X_g) + b_g X_g, X_g the activations' sum over group g: s and b are exact in bf16, X is taken in three
//    bf16 parts, so both terms are a few small MMAs per eight groups (and X itself a product with ones).  (fp32 sums of 64 products of magnitude 128 |x|: their
//    rounding stays below 1e-5 of the result.)
//  * Sorted rows: a CTA owns TM consecutive rows of the sorted list and runs one pass over K per expert it finds there; no tables.
//    With few rows per expert these passes would follow one another in a few CTAs: then a CTA owns one piece, up to TM rows of one
//    expert (cut where the expert changes and at multiples of TM), which it finds by counting the cuts of the list.
#include <type_traits>

#include "kernels.h"
#include "stream_ptx.cuh"

namespace qb {
namespace {

constexpr int kThreads = 256, kRing = 4;

struct TileK {
  const uint16_t* x; const uint32_t* w; const uint16_t* s; const uint16_t* b; uint16_t* y;
  int M, N, K, gshift;           // gshift 1: group size 128, every scale serves two 64-groups
  int64_t ldx, ldw, lds, ldy;
  // sorted rows: expert of row i, element strides between experts
  const void* rhs; int rhs_i64;
  int64_t wes, ses;
  int E;
  int pieces;                    // a CTA per piece of up to TM rows of one expert, instead of per TM rows of the list
};

template <int BITS, int GS, int TM, int WN>
struct Geo {
  static constexpr int TN = 32 * WN, WM = kThreads / 32 / WN, NT = TM / WM / 8;   // rows per tile; warps over tokens; n8 tiles per warp
  static constexpr int H = GS == 32 ? 2 : 1;                           // scale groups per 64 k
  static constexpr int BS = 8 / H;                                     // stages per block of 8 groups
  static constexpr int WROW = 64 * BITS / 8;                           // code bytes of a row and stage
  static constexpr int RAW = TM * 128, W = TN * WROW;
  static constexpr int XB = 3 * TM * 16, SB = TN * 16;                 // a block's activation sums [part][token][8]; scales (or biases) [row][8]
  static constexpr int OUTP = TN + 8;                                  // pitch of the output tile in shared memory
  static constexpr size_t kMain = (size_t)kRing * (RAW + W) + 2 * XB + 4 * SB;
  static constexpr int PARTP = TN + 4;                                 // pitch of the fp32 partial sums there
  static constexpr size_t kOut = (size_t)TM * PARTP * 4;
  static constexpr size_t kSmem = kMain > kOut ? kMain : kOut;
  static_assert(NT >= 1 && NT * WM * 8 == TM, "tile");
};

// 4 bits: A operands (pairs of codes i, i + 4 of the word) of two MMA steps as 128 + c
__device__ __forceinline__ void expand4(uint32_t w, uint32_t (&o)[4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) o[i] = lop3_and_or(w >> (4 * i), 0x000F000Fu, 0x43004300u);
}

// 8 bits: the pairs (0, 2) and (1, 3) of the word as integers 0..255
__device__ __forceinline__ uint32_t byte_pair(uint32_t v) {
  const __nv_bfloat162 r = bf16_of_bytes(v);
  return *(const uint32_t*)&r;
}

// GS: 32, or 64 (64 and 128)
template <int BITS, int GS, int TM, int WN, bool GROUPED>
__global__ void __launch_bounds__(kThreads, 2) qmm_tile_kernel(const __grid_constant__ TileK p) {
  using GE = Geo<BITS, GS, TM, WN>;
  constexpr int TN = GE::TN, WM = GE::WM, NT = GE::NT, H = GE::H;
  extern __shared__ __align__(128) unsigned char smem[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int wn = warp % WN, wm = warp / WN;
  const int n0 = blockIdx.x * TN;
  const uint32_t s0 = (uint32_t)__cvta_generic_to_shared(smem);
  unsigned char* raw_p = smem;
  unsigned char* w_p = raw_p + kRing * GE::RAW;
  unsigned char* xb_p = w_p + kRing * GE::W;                   // [2][part][token][8] bf16
  unsigned char* sb_p = xb_p + 2 * GE::XB;                     // [2][scales | biases][row][8] bf16
  const uint32_t raw_s = s0, w_s = s0 + kRing * GE::RAW;
  const int nst_all = (p.K + 63) / 64, ngrp = GS == 32 ? p.K / 32 : nst_all;   // scale groups (group size 128: each counts twice)
  // the stages of this CTA: all, or its share where a cluster splits K (blocks of 8 groups count from its first stage)
  const int nsplit = GROUPED ? 1 : (int)gridDim.z, rank = GROUPED ? 0 : (int)blockIdx.z;
  const int st0 = (int)((int64_t)nst_all * rank / nsplit), nst = (int)((int64_t)nst_all * (rank + 1) / nsplit) - st0;
  auto expert_of = [&](int row) -> int {
    return p.rhs_i64 ? (int)((const long long*)p.rhs)[row] : ((const int*)p.rhs)[row];
  };

  int m0 = blockIdx.y * TM, mtile = p.M - m0 < TM ? p.M - m0 : TM;
  if (GROUPED && p.pieces) {
    // this CTA's piece is number blockIdx.y: every thread counts the cuts among its share of the rows, whoever owns it finds it
    int* cnt = (int*)smem;
    const int R = (p.M + kThreads - 1) / kThreads, r0 = tid * R < p.M ? tid * R : p.M, r1 = r0 + R < p.M ? r0 + R : p.M;
    int n = 0, prev = r0 > 0 && r0 < r1 ? expert_of(r0 - 1) : -1;
    for (int r = r0; r < r1; ++r) { const int e = expert_of(r); n += r % TM == 0 || e != prev; prev = e; }
    int sum = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const int v = __shfl_up_sync(0xffffffffu, sum, o); if (lane >= o) sum += v; }
    if (lane == 31) cnt[warp] = sum;
    if (tid == 0) cnt[kThreads / 32] = -1;
    __syncthreads();
    for (int w = 0; w < warp; ++w) sum += cnt[w];
    int left = (int)blockIdx.y - (sum - n);     // cuts of this thread before the piece
    if (left >= 0 && left < n) {
      int r = r0;
      prev = r0 > 0 ? expert_of(r0 - 1) : -1;
      for (; r < r1; ++r) { const int e = expert_of(r); if (r % TM == 0 || e != prev) { if (left == 0) break; --left; } prev = e; }
      cnt[kThreads / 32] = r;
    }
    __syncthreads();
    m0 = cnt[kThreads / 32];
    if (m0 < 0) return;                         // fewer pieces than CTAs
    const int end = m0 - m0 % TM + TM;          // (an expert's end before it ends the segment below)
    mtile = (end < p.M ? end : p.M) - m0;
  }
  for (int lo = 0; lo < mtile;) {
    // the tokens [lo, hi) of this tile share one weight matrix
    int hi = mtile, ex = 0;
    if constexpr (GROUPED) {
      ex = expert_of(m0 + lo);
      int a = lo + 1, b = mtile;     // the list is ascending: first row with another expert
      while (a < b) { const int m = (a + b) >> 1; if (expert_of(m0 + m) > ex) b = m; else a = m + 1; }
      hi = a;
    }
    if (GROUPED && (ex < 0 || ex >= p.E)) { if (p.pieces) return; lo = hi; continue; }   // padding rows are left untouched, as in every other form
    const uint32_t* wq = p.w + (int64_t)ex * p.wes;
    const uint16_t* sp = p.s + (int64_t)ex * p.ses;
    const uint16_t* bp = p.b + (int64_t)ex * p.ses;
    const int c_lo = GROUPED ? lo / 8 : 0, c_hi = GROUPED ? (hi + 7) / 8 : TM / 8;   // n8 tiles with tokens of this segment

    // ---- copies of one stage into its ring slot: this thread's pieces, the same rows in every stage ----
    constexpr int XP = (TM * 8 + kThreads - 1) / kThreads, PC = GE::WROW / 16, WP = (TN * PC + kThreads - 1) / kThreads;
    const uint16_t* xsrc[XP];
    const unsigned char* wsrc[WP];
    uint32_t xn[XP], wn_b[WP];           // 16, or 0 for rows that do not exist (zeros)
    bool xuse[XP];                       // rows of token tiles without tokens of this segment are not touched
#pragma unroll
    for (int j = 0; j < XP; ++j) {
      const int i = tid + j * kThreads, row = i >> 3;
      const bool ok = row >= lo && row < hi && (TM * 8 >= kThreads || i < TM * 8);
      xsrc[j] = p.x + (int64_t)(m0 + (ok ? row : lo)) * p.ldx + (i & 7) * 8 + st0 * 64;
      xn[j] = ok ? 16u : 0u;
      xuse[j] = (TM * 8 >= kThreads || i < TM * 8) && row >= c_lo * 8 && row < c_hi * 8;
    }
#pragma unroll
    for (int j = 0; j < WP; ++j) {
      const int i = tid + j * kThreads, row = i / PC;
      const bool ok = row < TN && n0 + row < p.N;
      wsrc[j] = (const unsigned char*)(wq + (int64_t)(ok ? n0 + row : 0) * p.ldw) + (i % PC) * 16 + st0 * GE::WROW;
      wn_b[j] = ok ? 16u : 0u;
    }
    const uint32_t xdst = raw_s + (tid >> 3) * 128 + (((tid & 7) ^ ((tid >> 3) & 1)) << 4), wdst = w_s + tid * 16;
    // this thread's pieces of x in the order of the codes' pairs
    auto permute = [&](int slot) {
#pragma unroll
      for (int j = 0; j < XP; ++j)
        if (xuse[j]) {
          uint4* q = (uint4*)(raw_p + (xdst - raw_s) + slot * GE::RAW + j * (kThreads / 8) * 128);
          const uint4 v = *q;
          if constexpr (BITS == 4) *q = make_uint4(__byte_perm(v.x, v.z, 0x5410), __byte_perm(v.x, v.z, 0x7632), __byte_perm(v.y, v.w, 0x5410), __byte_perm(v.y, v.w, 0x7632));
          else *q = make_uint4(__byte_perm(v.x, v.y, 0x5410), __byte_perm(v.x, v.y, 0x7632), __byte_perm(v.z, v.w, 0x5410), __byte_perm(v.z, v.w, 0x7632));
        }
    };
    int is_st = 0, is_slot = 0;
    auto issue = [&]() {
      if (is_st < nst) {
        // of the last stage half may lie behind K (group size 32)
        const bool tail = GS == 32 && (st0 + is_st + 1) * 64 > p.K;
#pragma unroll
        for (int j = 0; j < XP; ++j) {
          if (xuse[j]) cp_async16_z(xdst + is_slot * GE::RAW + j * (kThreads / 8) * 128, xsrc[j], tail && (tid & 7) >= 4 ? 0u : xn[j]);
          xsrc[j] += 64;
        }
#pragma unroll
        for (int j = 0; j < WP; ++j) {
          if (TN * PC % kThreads == 0 || tid + j * kThreads < TN * PC)
            cp_async16_z(wdst + is_slot * GE::W + j * kThreads * 16, wsrc[j], tail && ((tid + j * kThreads) % PC) * 2 >= PC ? 0u : wn_b[j]);
          wsrc[j] += GE::WROW;
        }
      }
      ++is_st;
      is_slot = is_slot + 1 == kRing ? 0 : is_slot + 1;
      cp_async_commit();
    };
    // scales and biases of a block of 8 groups; groups behind K count as 0
    constexpr int SPT = (TN * 8 + kThreads - 1) / kThreads;
    uint16_t sv[SPT], bv[SPT];
    auto load_sb = [&](int blk) {
#pragma unroll
      for (int i = 0; i < SPT; ++i) {
        const int e = tid + i * kThreads, row = e >> 3, gi = st0 * H + blk * 8 + (e & 7);
        sv[i] = bv[i] = 0;
        if (row < TN && n0 + row < p.N && gi < ngrp && gi < (st0 + nst) * H) {
          const int64_t o = (int64_t)(n0 + row) * p.lds + (gi >> p.gshift);
          sv[i] = __ldg(sp + o);
          bv[i] = __ldg(bp + o);
        }
      }
    };
    auto store_sb = [&](int blk) {
      uint16_t* d = (uint16_t*)(sb_p + (blk & 1) * 2 * GE::SB);
#pragma unroll
      for (int i = 0; i < SPT; ++i) {
        const int e = tid + i * kThreads;
        if (TN * 8 >= kThreads || e < TN * 8) { d[e] = sv[i]; d[e + TN * 8] = bv[i]; }
      }
    };
    // this lane's 16 codes of row `row` in stage slot `slot`
    auto codes = [&](int slot, int row, uint32_t (&w)[BITS / 2]) {
      const unsigned char* q = w_p + slot * GE::W + row * GE::WROW;
      if constexpr (BITS == 4 && GS != 32) { const uint2 a = *(const uint2*)(q + 8 * t); w[0] = a.x; w[1] = a.y; }
      else if constexpr (BITS == 4) { w[0] = *(const uint32_t*)(q + 4 * t); w[1] = *(const uint32_t*)(q + 16 + 4 * t); }
      else if constexpr (GS != 32) { const uint4 a = *(const uint4*)(q + 16 * t); w[0] = a.x; w[1] = a.y; w[2] = a.z; w[3] = a.w; }
      else { const uint2 a = *(const uint2*)(q + 8 * t), c = *(const uint2*)(q + 32 + 8 * t); w[0] = a.x; w[1] = a.y; w[2] = c.x; w[3] = c.y; }
    };

    float acc[2][NT][4];
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
      for (int n = 0; n < NT; ++n) acc[m][n][0] = acc[m][n][1] = acc[m][n][2] = acc[m][n][3] = 0.f;

    // the terms b X and -128 s X of a finished block
    auto finish_block = [&](int blk) {
      const unsigned char* sq = sb_p + (blk & 1) * 2 * GE::SB;
      const unsigned char* xq = xb_p + (blk & 1) * GE::XB;
      uint32_t sa[2][2], ba[2][2];
#pragma unroll
      for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int o = (wn * 32 + m * 16 + g + 8 * h) * 16 + 4 * t;
          sa[m][h] = *(const uint32_t*)(sq + o);
          ba[m][h] = *(const uint32_t*)(sq + GE::SB + o);
        }
#pragma unroll
      for (int n = 0; n < NT; ++n) {
        const int ct = wm * NT + n;
        if (GROUPED && (ct < c_lo || ct >= c_hi)) continue;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const uint32_t x = *(const uint32_t*)(xq + (k * TM + ct * 8 + g) * 16 + 4 * t);
#pragma unroll
          for (int m = 0; m < 2; ++m) mma_bf16_1688(acc[m][n], ba[m][0], ba[m][1], x);
          if constexpr (BITS == 4) {
            const __nv_bfloat162 x128 = __hmul2(*(const __nv_bfloat162*)&x, __float2bfloat162_rn(-128.f));   // exact
#pragma unroll
            for (int m = 0; m < 2; ++m) mma_bf16_1688(acc[m][n], sa[m][0], sa[m][1], *(const uint32_t*)&x128);
          }
        }
      }
    };

    __syncthreads();                  // the ring and the output tile of the segment before are no longer read
#pragma unroll
    for (int i = 0; i < kRing - 1; ++i) issue();
    for (int i = tid; i < 2 * GE::XB / 16; i += kThreads) ((uint4*)xb_p)[i] = make_uint4(0u, 0u, 0u, 0u);
    load_sb(0);
    store_sb(0);
    load_sb(1);
#pragma unroll 1
    for (int st = 0; st < nst; ++st) {
      cp_async_wait<kRing - 2>();     // stage st has landed (this thread's part)
      permute(st % kRing);
      __syncthreads();                // ... everybody's; slot st - 1 and, at a block's start, the block before are complete
      issue();
      const int blk = st / GE::BS, in = st % GE::BS;
      if (in == 0) {
        if (blk > 0) finish_block(blk - 1);
      } else if (in == 1 && st + GE::BS - 1 < nst) {   // (everybody is past finish_block: its buffer takes the next block)
        store_sb(blk + 1);
        load_sb(blk + 2);
      }
      const int slot = st % kRing;
      uint32_t A[2][4][4];
      float sc[2][2][H];              // [m tile][row g, g + 8][half]
#pragma unroll
      for (int m = 0; m < 2; ++m) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int row = wn * 32 + m * 16 + g + 8 * h;
          uint32_t w[BITS / 2];
          codes(slot, row, w);
          if constexpr (BITS == 4) {
#pragma unroll
            for (int q = 0; q < 2; ++q) {
              uint32_t o[4];
              expand4(w[q], o);
              A[m][2 * q][h] = o[0]; A[m][2 * q][2 + h] = o[1]; A[m][2 * q + 1][h] = o[2]; A[m][2 * q + 1][2 + h] = o[3];
            }
          } else {
#pragma unroll
            for (int k = 0; k < 4; ++k) { A[m][k][h] = byte_pair(w[k] & 0x00FF00FFu); A[m][k][2 + h] = byte_pair((w[k] >> 8) & 0x00FF00FFu); }
          }
          const uint16_t* sq = (const uint16_t*)(sb_p + (blk & 1) * 2 * GE::SB) + row * 8 + in * H;
#pragma unroll
          for (int k = 0; k < H; ++k) sc[m][h][k] = bf16_bits_to_f32(sq[k]);
        }
      }
#pragma unroll
      for (int n = 0; n < NT; ++n) {
        const int ct = wm * NT + n;     // token tile
        if (GROUPED && (ct < c_lo || ct >= c_hi)) continue;
        // this lane's 16 activations of token g, in the order of the codes
        const unsigned char* xr = raw_p + slot * GE::RAW + (ct * 8 + g) * 128;
        const int cA = GS == 32 ? t : 2 * t, cB = GS == 32 ? 4 + t : 2 * t + 1;
        const uint4 q0 = *(const uint4*)(xr + ((cA ^ (g & 1)) << 4)), q1 = *(const uint4*)(xr + ((cB ^ (g & 1)) << 4));
        const uint32_t bb[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
#pragma unroll
        for (int h = 0; h < H; ++h) {
          float d[2][4];
#pragma unroll
          for (int k = 4 * h / H; k < 4 * (h + 1) / H; ++k)
#pragma unroll
            for (int m = 0; m < 2; ++m) {
              if (k == 4 * h / H) mma_bf16_16816_z(d[m], A[m][k], bb[2 * k], bb[2 * k + 1]);
              else mma_bf16_16816(d[m], A[m][k], bb[2 * k], bb[2 * k + 1]);
            }
#pragma unroll
          for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[m][n][i] = fmaf(sc[m][i >> 1][h], d[m][i], acc[m][n][i]);
          // group sums of this token tile: a product with ones, by one of the warps that hold its fragments
          if (n % WN == wn) {
            const uint32_t ones[4] = {0x3F803F80u, 0x3F803F80u, 0x3F803F80u, 0x3F803F80u};
            float x[4];
#pragma unroll
            for (int k = 4 * h / H; k < 4 * (h + 1) / H; ++k) {
              if (k == 4 * h / H) mma_bf16_16816_z(x, ones, bb[2 * k], bb[2 * k + 1]);
              else mma_bf16_16816(x, ones, bb[2 * k], bb[2 * k + 1]);
            }
            // every row of the product is the same: the lanes of row k store part k of tokens 2t, 2t + 1
            uint16_t h0 = 0, h1 = 0;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
              if (k <= g) { h0 = f32_to_bf16_bits(x[0]); h1 = f32_to_bf16_bits(x[1]); }
              x[0] -= bf16_bits_to_f32(h0); x[1] -= bf16_bits_to_f32(h1);
            }
            uint16_t* q = (uint16_t*)(xb_p + (blk & 1) * GE::XB + (g * TM + ct * 8 + 2 * t) * 16) + in * H + h;
            if (g < 3) { q[0] = h0; q[8] = h1; }
          }
        }
      }
    }
    __syncthreads();
    finish_block((nst - 1) / GE::BS);
    cp_async_wait<0>();
    __syncthreads();
    const int nv = p.N - n0 < TN ? p.N - n0 : TN;
    const bool vec = ((((uintptr_t)p.y) | (uintptr_t)(p.ldy * 2)) & 15) == 0;
    if constexpr (!GROUPED) {
      if (nsplit > 1) {
        // fp32 partial sums to shared memory; every CTA of the cluster adds up its share of the tile's rows, in rank order
        float* part = (float*)smem;
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
          for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int i = 0; i < 4; ++i)
              part[((wm * NT + n) * 8 + 2 * t + (i & 1)) * GE::PARTP + wn * 32 + m * 16 + g + 8 * (i >> 1)] = acc[m][n][i];
        cluster_sync_all();
        const int r0 = mtile * rank / nsplit, r1 = mtile * (rank + 1) / nsplit;
        for (int i = r0 * (TN / 4) + tid; i < r1 * (TN / 4); i += kThreads) {
          const int row = i / (TN / 4), c = (i % (TN / 4)) * 4;
          const uint32_t at = s0 + (row * GE::PARTP + c) * 4;
          float4 v = ld_cluster_f32x4(map_to_rank(at, 0));
          for (int r = 1; r < nsplit; ++r) {
            const float4 q = ld_cluster_f32x4(map_to_rank(at, (uint32_t)r));
            v.x += q.x; v.y += q.y; v.z += q.z; v.w += q.w;
          }
          uint16_t* yr = p.y + (int64_t)(m0 + row) * p.ldy + n0 + c;
          if (vec && c + 4 <= nv) *(uint2*)yr = make_uint2(pack2(v.x, v.y), pack2(v.z, v.w));
          else {
            const float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int k = 0; k < 4; ++k)
              if (c + k < nv) yr[k] = f32_to_bf16_bits(e[k]);
          }
        }
        cluster_sync_all();   // the peers' shared memory stays alive until everybody has read it
        return;
      }
    }
    // ---- the tile as bf16 through shared memory, rows of y in whole pieces ----
    uint16_t* so = (uint16_t*)smem;
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i)
          so[((wm * NT + n) * 8 + 2 * t + (i & 1)) * GE::OUTP + wn * 32 + m * 16 + g + 8 * (i >> 1)] = f32_to_bf16_bits(acc[m][n][i]);
    __syncthreads();
    for (int i = lo * (TN / 8) + tid; i < hi * (TN / 8); i += kThreads) {
      const int row = i / (TN / 8), c = (i % (TN / 8)) * 8;
      uint16_t* yr = p.y + (int64_t)(m0 + row) * p.ldy + n0 + c;
      const uint16_t* sr = so + row * GE::OUTP + c;
      if (vec && c + 8 <= nv) *(uint4*)yr = *(const uint4*)sr;
      else
        for (int k = 0; k < 8; ++k)
          if (c + k < nv) yr[k] = sr[k];
    }
    if (GROUPED && p.pieces) return;
    lo = hi;
  }
}

template <int BITS, int GS, int TM, int WN, bool GROUPED = false>
cudaError_t launch_inst(const TileK& p, int nsplit, cudaStream_t st) {
  using GE = Geo<BITS, GS, TM, WN>;
  static_assert(GE::kSmem <= 227 * 1024, "shared memory");
  auto kern = qmm_tile_kernel<BITS, GS, TM, WN, GROUPED>;
  static bool done[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  {
    std::lock_guard<std::mutex> lk(setup_mutex());   // first use on a device, from any thread
    if (dev < 0 || dev >= 64 || !done[dev]) {
      const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GE::kSmem);
      if (e != cudaSuccess) return e;
      if (dev >= 0 && dev < 64) done[dev] = true;
    }
  }
  const dim3 grid((unsigned)((p.N + GE::TN - 1) / GE::TN), (unsigned)(p.pieces ? p.pieces : (p.M + TM - 1) / TM), (unsigned)nsplit);
  if (nsplit == 1) return launch_kernel(kern, grid, dim3(kThreads), GE::kSmem, st, p);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = GE::kSmem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = (unsigned)nsplit;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const cudaError_t e = launch_clusters(cfg, kern, p);
  if (e == cudaSuccess) return e;
  (void)cudaGetLastError();   // a cluster this launch could not place: a CTA takes the whole of K
  return launch_kernel(kern, dim3(grid.x, grid.y), dim3(kThreads), GE::kSmem, st, p);
}
template <int BITS, int GS>
cudaError_t launch_shape(const TileK& p, int tm, int nsplit, cudaStream_t st) {
  if (p.rhs) return tm == 32 ? launch_inst<BITS, GS, 32, 4, true>(p, 1, st) : launch_inst<BITS, GS, 64, 4, true>(p, 1, st);
  if (tm == 32) return launch_inst<BITS, GS, 32, 4, false>(p, nsplit, st);
  return tm == 64 ? launch_inst<BITS, GS, 64, 4, false>(p, nsplit, st) : launch_inst<BITS, GS, 128, 2, false>(p, nsplit, st);
}
template <int BITS>
cudaError_t launch_gs(const TileK& p, int gs, int tm, int nsplit, cudaStream_t st) {
  return gs == 32 ? launch_shape<BITS, 32>(p, tm, nsplit, st) : launch_shape<BITS, 64>(p, tm, nsplit, st);
}

// Tile of a dense product and shares of K: the time of a CTA is its stages x the time of a stage (alone on its SM / with a second
// CTA there) plus about 4.5 us of launch, first copies and store, and 1.5 us for the cluster's sum; an SM runs two CTAs at a time,
// clusters of three to eight leave up to an eighth of the places empty.  (us; within 20 % of the measured times over 5 - 700 CTAs
// and 2 - 200 stages)
void pick_tile(int64_t M, int64_t N, int64_t nst, int* tm, int* nsplit) {
  struct Cand { int tm, tn; double one, two; };
  static const Cand cand[3] = {{64, 128, 0.98, 1.39}, {128, 64, 1.17, 1.6}, {32, 128, 0.64, 0.95}};
  double best = -1.0;
  for (const Cand& c : cand)
    for (int s = 1; s <= 8 && s <= nst; ++s) {
      const int64_t clusters = ((N + c.tn - 1) / c.tn) * ((M + c.tm - 1) / c.tm), cap = (int64_t)(2 * sm_count() * (s > 2 ? 0.87 : 1.0) / s);
      const int64_t full = clusters / cap, rem = clusters % cap;
      const double stages = (double)nst / s, fixed = s > 1 ? 6.0 : 4.5;
      const double cost = full * (stages * c.two + fixed) + (rem == 0 ? 0.0 : stages * (2 * rem <= cap ? c.one : c.two) + fixed);
      if (best < 0.0 || cost < best - 1e-9) { best = cost; *tm = c.tm; *nsplit = s; }
    }
}
bool format_ok(int bits, int gs, int64_t K) {
  return (bits == 4 || bits == 8) && (gs == 32 || gs == 64 || gs == 128) && K > 0 && K % gs == 0 && K <= (1 << 24);
}

}  // namespace

bool qmm_tile_supported(const QmmArgs& a) {
  if (!a.transpose || a.nbatch != 1 || a.x_dtype != QB200_BFLOAT16 || !format_ok(a.bits, a.gs, a.K)) return false;
  if (a.M < 1 || a.M > 32 * 65535 || a.N < 1 || a.N > (1 << 24)) return false;
  if (((uintptr_t)a.x & 15) || a.ldx % 8 != 0 || ((uintptr_t)a.w & 15) || a.ldw % 4 != 0) return false;
  return true;
}
cudaError_t launch_qmm_tile(const QmmArgs& a, cudaStream_t st) {
  TileK p = {};
  p.x = (const uint16_t*)a.x + a.xb.offset(0); p.w = a.w + a.wb.offset(0);
  p.s = (const uint16_t*)a.s + a.sb.offset(0); p.b = (const uint16_t*)a.b + a.sb.offset(0); p.y = (uint16_t*)a.y + a.yb.offset(0);
  p.gshift = a.gs == 128 ? 1 : 0;
  p.M = (int)a.M; p.N = (int)a.N; p.K = (int)a.K; p.ldx = a.ldx; p.ldw = a.ldw; p.lds = a.lds; p.ldy = a.ldy;
  int tm = 64, nsplit = 1;
  pick_tile(a.M, a.N, (a.K + 63) / 64, &tm, &nsplit);
  return a.bits == 4 ? launch_gs<4>(p, a.gs, tm, nsplit, st) : launch_gs<8>(p, a.gs, tm, nsplit, st);
}

bool gather_tile_supported(const GatherArgs& a) {
  if (!a.sorted || a.lhs != nullptr || a.M != 1 || a.XB != a.I || a.w2 || a.x_dtype != QB200_BFLOAT16 || !format_ok(a.bits, a.gs, a.K)) return false;
  for (int d = 0; d < a.xbcast.nd; ++d)
    if (a.xbcast.shape[d] != 1 && a.xbcast.stride[d] == 0) return false;   // one activation row per output row, in order
  if (a.I < 1 || a.I > 32 * 65535 || a.N < 1 || a.N > (1 << 24) || a.E < 1 || a.E > (1 << 20)) return false;
  if (((uintptr_t)a.x & 15) || a.K % 8 != 0 || ((uintptr_t)a.w & 15) || (a.K * a.bits / 32) % 4 != 0 || a.w_expert_stride % 4 != 0) return false;
  return true;
}
cudaError_t launch_gather_tile(const GatherArgs& a, cudaStream_t st) {
  TileK p = {};
  p.x = (const uint16_t*)a.x; p.w = a.w; p.s = (const uint16_t*)a.s; p.b = (const uint16_t*)a.b; p.y = (uint16_t*)a.y;
  p.gshift = a.gs == 128 ? 1 : 0;
  p.M = (int)a.I; p.N = (int)a.N; p.K = (int)a.K; p.ldx = a.K; p.ldw = a.K * a.bits / 32; p.lds = a.K / a.gs; p.ldy = a.N;
  p.rhs = a.rhs; p.rhs_i64 = a.rhs_dtype == QB200_INT64; p.wes = a.w_expert_stride; p.ses = a.s_expert_stride; p.E = (int)a.E;
  // Tokens per tile by the rows an expert has on average.  A CTA per piece while finding it is quick and tiles hold several
  // experts (us, per tile -> per piece: 96 rows, 64 experts, 2048 x 896 163 -> 41; 200 rows, 8 experts, 1024 x 640, 8 bits
  // 23 -> 14; 968 rows, 64 experts, 1792 x 896 83 -> 73; but 4800 rows, 64 experts, 1024 x 640 74 -> 84).
  const int tm = a.I / a.E > 32 ? 64 : 32;
  if (a.I <= 4096) p.pieces = (int)((a.I + tm - 1) / tm + (a.E < a.I ? a.E : a.I) - 1);
  return a.bits == 4 ? launch_gs<4>(p, a.gs, tm, 1, st) : launch_gs<8>(p, a.gs, tm, 1, st);
}

}  // namespace qb
