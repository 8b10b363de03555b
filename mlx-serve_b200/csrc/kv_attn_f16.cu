// Split-KV flash-decode over the affine-quantized KV cache: head dim 64 or 128, group size 64, 4- or 8-bit codes,
// up to 8 query heads per cache head and up to 8 query positions, on the fp16 tensor cores.
//
// Semantics: kv_quant.quantAttention at T_q == 1 (mlx-serve src/kv_quant.zig:478-687) with K/V kept in fp32 (q*s+b)
// exactly as the packed decode kernel does (src/transformer.zig:4890-5006); the verify widths' causal tail
// (src/transformer.zig:5314-5318); per-sequence lengths as the batched path's additive mask
// (src/transformer.zig:10216-10249); partials merged as src/transformer.zig:5194-5203.
//
// Organisation (HBM-bound by bytes: the packed codes are read once, straight from the strided cache views; what a kernel
// of this kind runs out of in long batches is issue slots, so the arithmetic is arranged around spending few of them per code):
//  * grid (split, kv head x query tile, sequence); 4 warps per CTA, three CTAs per SM.  A warp walks blocks of 64
//    tokens with its own online softmax and its own cp.async ring, so no warp waits on another for data.
//  * A code c (up to 8 bits) in the low bits of a 16-bit word IS the fp16 subnormal c * 2^-24, exactly: one AND turns a
//    packed word into an MMA operand register (two codes), with no conversion, no offset to cancel and no rounding.
//    The nibble next to it is 16 * c * 2^-24; its partner operand, or the output column, carries the 1/16.
//  * Query rows are the 16 rows of the A operand: 8 queries (a query tile), and in rows 8..15 the low-order parts of the
//    same 8 rows -- of the queries when they are fp32, and of the probabilities always -- so that hi + lo gives 22
//    significant bits for the rows that an 8-query tile would leave empty.  More than 8 queries run as more tiles, which
//    read the cache again out of L2.
//  * Scores: K codes are the B operand (8 tokens x 16 dims).  Scale per (token, 64-group) multiplies the fp32 sums; the
//    bias term is one more MMA, biases against the group sums of q in three bf16 parts.
//  * Values: the probabilities are already laid out as the A operand of P.V (the rows of a score tile are the rows of
//    the next product), multiplied in fp32 by the V scale of (token, group).  The V codes become the B operand through
//    ldmatrix.m16n16.trans.b8, which hands each lane four tokens of one byte column: AND and shift give pairs of tokens
//    of one dim.  The V bias term is a plain fp32 dot of p with the biases.
//  * The running reference r of the softmax (p = 2^(s - r)) is kept below the block maximum by the exponent of the
//    block's largest V scale, so p * v_scale uses fp16's range from the top whatever the scales are.
// Bound: the latency of a warp's chain of dependent instructions, with few warps to hide it.  408 warp instructions per 16 tokens at
// 4 bits and head dim 128; IPC 2.1 with 12 warps on an SM (long batches), 1.5 - 1.6 with the 7 - 9 that short ones leave there (ncu).
// What it replaces and when it runs: the launch rule in kv_attn.cu.
#include <mutex>

#include <type_traits>

#include "kernels.h"
#include "stream_ptx.cuh"

namespace qb {
namespace {

constexpr int kWarps = 4;
constexpr int kBlk = 64;              // tokens per softmax block
constexpr int kHalf = 32;             // tokens per ring stage
constexpr int kRows = 8;              // queries per tile
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kNegBig = -1e30f;

template <int BITS, int D> struct Geo {
  static constexpr int G = D / 64;                        // scale groups per token
  static constexpr int ROWB = D * BITS / 8;               // code bytes per token
  static constexpr int CH = ROWB / 16;                    // 16-byte chunks per token
  static constexpr int STAGE = kHalf * ROWB;              // bytes of one ring stage (32 tokens of K or of V)
  static constexpr int STAGES = STAGE > 2048 ? 3 : 4;      // 3 x 4 KB keeps three CTAs on an SM; the scales' lookahead needs <= 4
  static constexpr int SB = kBlk * G * 2;                 // bytes of one of {ks, kb, vs, vb} for a block
  static constexpr int RING = STAGES * STAGE;
  static constexpr int NT = D / 8;                        // n8 tiles of the output
};
template <int BITS, int D> constexpr size_t smem_bytes() {
  using G = Geo<BITS, D>;
  const size_t main = (size_t)kWarps * (G::RING + 2 * 4 * G::SB) + G::G * 4 * 32 * 16 + kRows * 32;
  const size_t merge = (size_t)(kWarps + 1) * kRows * (D + 2) * 4;   // the ring is reused for the merge
  return main > merge ? main : merge;
}

struct F16K {
  KvAttnArgs a;
  int nsplit;
  int gqa, nq;     // query heads per cache head; queries per (sequence, cache head) = gqa * T_q
  int qtiles;
  int fused;       // the splits of a (sequence, kv head, tile) are the CTAs of one cluster, which merges and stores
  float* part_m; float* part_l; float* part_o;
};

// 16-byte chunk swizzle of a stage row: the score phase reads 8 consecutive rows, the value phase rows {0,8,1,9,..}; with
// this both take the fewest shared-memory wavefronts at every row size.
template <int CH> __device__ __forceinline__ int swz(int row) {
  int f = (row >> 3) & 1;
  if (CH >= 4) f |= ((row >> 1) & 1) << 1;
  if (CH >= 8) f |= (row & 1) << 2;
  return f;
}
// x = hi + lo: hi is x with the mantissa cut to fp16's, lo the exact rest; both packed in pairs (a in the low half)
__device__ __forceinline__ void split2(float a, float b, uint32_t& hi, uint32_t& lo) {
  const float ah = __uint_as_float(__float_as_uint(a) & 0xFFFFE000u), bh = __uint_as_float(__float_as_uint(b) & 0xFFFFE000u);
  hi = pack_f16x2(ah, bh);
  lo = pack_f16x2(a - ah, b - bh);
}

// TAB = KvSeqTable: sequence b reads its own cache view from the table; KvNoTable: one strided [B, Hkv, T, .] tensor.
template <int BITS, int D, bool QF32, class TAB>
__global__ void __launch_bounds__(kWarps * 32, 3) kv_f16_kernel(F16K p, const __grid_constant__ TAB tab) {
  constexpr bool PTRS = std::is_same<TAB, KvSeqTable>::value;
  using GE = Geo<BITS, D>;
  constexpr int G = GE::G, CH = GE::CH;
  extern __shared__ __align__(128) unsigned char smem[];
  const KvAttnArgs& a = p.a;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int split = blockIdx.x, hk = blockIdx.y / p.qtiles, qt = blockIdx.y - hk * p.qtiles;
  const int64_t b = blockIdx.z;

  unsigned char* ring = smem;
  unsigned char* sbbuf = ring + (size_t)kWarps * GE::RING;
  uint2* qfrag = (uint2*)(sbbuf + (size_t)kWarps * 2 * 4 * GE::SB);   // [step][hi | lo][lane]: (a0, a2)
  float* qc = (float*)(qfrag + G * 4 * 2 * 32);                       // [8]: factor of row r's scores
  uint32_t* qbias = (uint32_t*)(qc + kRows);                          // [8][3]: bias-MMA operand of row r

  // ---- this sequence's cache view ----
  const unsigned char* kq_base; const unsigned char* vq_base;
  const uint16_t* sbase[4];   // ks, kb, vs, vb
  int64_t kq_tok, ksb_tok, vq_tok, vsb_tok, T_seq;
  if constexpr (PTRS) {
    const KvSeq& q = tab.s[b];
    kq_base = (const unsigned char*)(q.kq + hk * q.kq_str[0]);
    vq_base = (const unsigned char*)(q.vq + hk * q.vq_str[0]);
    sbase[0] = (const uint16_t*)q.ks + hk * q.ksb_str[0]; sbase[1] = (const uint16_t*)q.kb + hk * q.ksb_str[0];
    sbase[2] = (const uint16_t*)q.vs + hk * q.vsb_str[0]; sbase[3] = (const uint16_t*)q.vb + hk * q.vsb_str[0];
    kq_tok = q.kq_str[1]; ksb_tok = q.ksb_str[1]; vq_tok = q.vq_str[1]; vsb_tok = q.vsb_str[1];
    T_seq = q.T;
  } else {
    kq_base = (const unsigned char*)(a.kq + b * a.kq_str[0] + hk * a.kq_str[1]);
    vq_base = (const unsigned char*)(a.vq + b * a.vq_str[0] + hk * a.vq_str[1]);
    const int64_t ko = b * a.ksb_str[0] + hk * a.ksb_str[1], vo = b * a.vsb_str[0] + hk * a.vsb_str[1];
    sbase[0] = (const uint16_t*)a.ks + ko; sbase[1] = (const uint16_t*)a.kb + ko;
    sbase[2] = (const uint16_t*)a.vs + vo; sbase[3] = (const uint16_t*)a.vb + vo;
    kq_tok = a.kq_str[2]; ksb_tok = a.ksb_str[2]; vq_tok = a.vq_str[2]; vsb_tok = a.vsb_str[2];
    T_seq = a.T;
  }
  int64_t len = a.kv_lens ? (int64_t)a.kv_lens[b] : T_seq;
  len = len > T_seq ? T_seq : (len < 0 ? 0 : len);
  // every sequence is cut into nsplit parts by its own length, so that ragged batches stay balanced
  const int64_t tps = ((len + p.nsplit - 1) / p.nsplit + kBlk - 1) / kBlk * kBlk;
  const int64_t t_begin = (int64_t)split * tps;
  int64_t t_end = t_begin + tps;
  t_end = t_end > len ? len : t_end;
  const int nblocks = t_end > t_begin ? (int)((t_end - t_begin + kBlk - 1) / kBlk) : 0;
  const int my_blocks = warp < nblocks ? (nblocks - warp + kWarps - 1) / kWarps : 0;
  const int my_items = my_blocks * 4;   // per block: two K stages, two V stages
  const int n_tok = nblocks ? (int)(t_end - t_begin) : 0;   // tokens of this split; positions below are relative to t_begin

  // ---- producer ----
  const uint32_t my_ring = (uint32_t)__cvta_generic_to_shared(ring + (size_t)warp * GE::RING);
  const unsigned char* my_ring_p = ring + (size_t)warp * GE::RING;
  constexpr int RPI = 32 / CH;                          // token rows covered by one copy instruction
  const int cc = lane % CH, r0 = lane / CH;
  auto issue = [&](int item, int stage) {
    const int tok0 = (warp + (item >> 2) * kWarps) * kBlk + (item & 1) * kHalf;
    const bool isv = (item & 2) != 0;
    const int64_t cstr = (isv ? vq_tok : kq_tok) * 4;
    const unsigned char* src = (isv ? vq_base : kq_base) + (t_begin + tok0 + r0) * cstr + cc * 16;
    const uint32_t st = my_ring + stage * GE::STAGE;
#pragma unroll
    for (int r = 0; r < kHalf / RPI; ++r) {
      const int row = r0 + r * RPI;
      // tokens behind the split's end are not read: their codes become 0
      cp_async16_z(st + row * GE::ROWB + ((cc ^ swz<CH>(row)) << 4), src + r * RPI * cstr, tok0 + row < n_tok ? 16u : 0u);
    }
  };
  // scales and biases of a block: [ks, kb, vs, vb][64 tokens][G], zero behind the split's end
  unsigned char* my_sb_p = sbbuf + (size_t)warp * 2 * 4 * GE::SB;
  const uint32_t my_sb = (uint32_t)__cvta_generic_to_shared(my_sb_p);
  bool vec = ksb_tok == G && vsb_tok == G;              // rows packed and 16-byte aligned: vector copies
#pragma unroll
  for (int i = 0; i < 4; ++i) vec = vec && (((uintptr_t)(sbase[i] + t_begin * G)) & 15) == 0;
  auto issue_sb = [&](int bi) {
    const int tok0 = (warp + bi * kWarps) * kBlk;
    const uint32_t dst0 = my_sb + (bi & 1) * 4 * GE::SB;
    if (vec) {
      constexpr int PC = GE::SB / 16;                   // 16-byte pieces per array: 8 G
#pragma unroll
      for (int i = lane; i < 4 * PC; i += 32) {
        const int arr = i / PC, pc = i - arr * PC;
        const int left = (n_tok - tok0) * G * 2 - pc * 16;
        const uint16_t* base = arr == 0 ? sbase[0] : (arr == 1 ? sbase[1] : (arr == 2 ? sbase[2] : sbase[3]));
        cp_async16_z(dst0 + arr * GE::SB + pc * 16, base + (t_begin + tok0) * G + pc * 8, left >= 16 ? 16u : (left > 0 ? (uint32_t)left : 0u));
      }
    } else {
      uint16_t* dst = (uint16_t*)(my_sb_p + (bi & 1) * 4 * GE::SB);
#pragma unroll
      for (int arr = 0; arr < 4; ++arr) {
        const int64_t str = arr < 2 ? ksb_tok : vsb_tok;
        uint16_t v[2][G];
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int c = 0; c < G; ++c) {
            const int tok = tok0 + h * 32 + lane;
            v[h][c] = tok < n_tok ? sbase[arr][(t_begin + tok) * str + c] : (uint16_t)0;
          }
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int c = 0; c < G; ++c) dst[arr * (GE::SB / 2) + (h * 32 + lane) * G + c] = v[h][c];
      }
    }
  };
  if (my_blocks > 0) issue_sb(0);
  int issued = 0;
#pragma unroll
  for (int i = 0; i < GE::STAGES - 1; ++i) {
    if (issued < my_items) issue(issued, issued % GE::STAGES);
    cp_async_commit();
    ++issued;
  }

  // ---- stage the queries: 8 rows as A fragments, hi and lo ----
  // One thread per (row, 8 consecutive dims); the D / 8 threads of a row are neighbours in a warp.
  {
    constexpr int TPR = D / 8;
    const int row = tid / TPR, c = tid % TPR, r = qt * kRows + row;
    const bool live = row < kRows && r < p.nq;
    float f[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] = 0.f;
    if (live) {
      const int tq = r / p.gqa, h = r - tq * p.gqa;
      const int64_t off = b * a.q_str[0] + (int64_t)(hk * p.gqa + h) * a.q_str[1] + tq * a.q_tq + c * 8;
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] = QF32 ? ((const float*)a.q)[off + j] : bf16_bits_to_f32(((const uint16_t*)a.q)[off + j]);
    }
    float mx = 0.f, sum = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) { mx = fmax_nan(mx, fabsf(f[j])); sum += f[j]; }
#pragma unroll
    for (int o = 1; o < TPR; o <<= 1) mx = fmax_nan(mx, __shfl_xor_sync(0xffffffffu, mx, o));
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);   // over a 64-group
    int e = (int)((__float_as_uint(mx) >> 23) & 0xFF) - 127;    // mx < 2^(e + 1)
    e = e < -100 ? -100 : (e > 110 ? 110 : e);
    const float up = pow2i(14 - e);
    if (row < kRows) {
      const int tt = (c >> 1) & 3, jm = c & 1, grp = c >> 3;
      if (c == 0) qc[row] = poison_if(nonfinite(mx), pow2i(24 - 14 + e) * (a.scale * kLog2e));
      if ((c & 7) == 0) {
        // s = qc * (scale * sum q~ c 2^-24 + bias * sum q~ 2^-24): the sum in three bf16 parts
        float v = sum * up * 5.9604644775390625e-8f;
        uint16_t parts[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) { parts[i] = f32_to_bf16_bits(v); v -= bf16_bits_to_f32(parts[i]); }
        uint16_t* d = (uint16_t*)(qbias + row * 3);
        if (G == 2) { d[grp] = parts[0]; d[2 + grp] = parts[1]; d[4 + grp] = parts[2]; }
        else { d[0] = parts[0]; d[1] = parts[1]; d[2] = parts[2]; d[3] = 0; d[4] = 0; d[5] = 0; }
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] *= up;
      // word jm of this lane quarter's two (4-bit) or words 2jm, 2jm + 1 of its four (8-bit): two MMA steps
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float v0, v1, v2, v3;
        if constexpr (BITS == 4) { v0 = f[2 * h]; v1 = f[2 * h + 4]; v2 = f[2 * h + 1] * 0.0625f; v3 = f[2 * h + 5] * 0.0625f; }
        else { v0 = f[4 * h]; v1 = f[4 * h + 2]; v2 = f[4 * h + 1]; v3 = f[4 * h + 3]; }
        uint2 hi, lo;
        if constexpr (QF32) { split2(v0, v1, hi.x, lo.x); split2(v2, v3, hi.y, lo.y); }
        else { hi = make_uint2(pack_f16x2(v0, v1), pack_f16x2(v2, v3)); lo = make_uint2(0u, 0u); }
        uint2* d = qfrag + (size_t)((grp * 4 + jm * 2 + h) * 2) * 32 + row * 4 + tt;
        d[0] = hi;
        if constexpr (QF32) d[32] = lo;
      }
    }
  }
  __syncthreads();
  uint2 qf[G * 4];                                  // hi fragments stay in registers, lo ones are read as they are needed
#pragma unroll
  for (int i = 0; i < G * 4; ++i) qf[i] = qfrag[(size_t)i * 64 + lane];
  const uint2* qlo = qfrag + 32 + lane;
  const float C = qc[g];
  const uint32_t qb = t < 3 ? qbias[g * 3 + t] : 0u;
  // causal tail: query position tq of a tile's row g sees the first len - T_q + 1 + tq tokens
  const int my_lim = (int)(len - t_begin) - (a.Tq - 1) + (qt * kRows + g) / p.gqa;
  const int lim = my_lim < n_tok ? my_lim : n_tok;

  int consumed = 0;
  auto acquire = [&]() -> const unsigned char* {
    if (issued < my_items) issue(issued, issued % GE::STAGES);
    cp_async_commit();
    ++issued;
    cp_async_wait<GE::STAGES - 1>();
    __syncwarp();
    const unsigned char* st = my_ring_p + (consumed % GE::STAGES) * GE::STAGE;
    ++consumed;
    return st;
  };

  float r_run = kNegBig, l_part = 0.f;
  float O[GE::NT][4];
  float ob[G];
#pragma unroll
  for (int i = 0; i < GE::NT; ++i) O[i][0] = O[i][1] = O[i][2] = O[i][3] = 0.f;
#pragma unroll
  for (int i = 0; i < G; ++i) ob[i] = 0.f;

  for (int bi = 0; bi < my_blocks; ++bi) {
    const int tok_blk = (warp + bi * kWarps) * kBlk;
    const unsigned char* sbb = my_sb_p + (bi & 1) * 4 * GE::SB;
    if (bi + 1 < my_blocks) issue_sb(bi + 1);   // joins the copy group of this block's first acquire
    float sc[16];       // scores (log2 domain) of row g; slot 4 * sub + 2 * j + i = token 16 * sub + 8 * j + 2 * t + i
    // ---------------- scores ----------------
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const unsigned char* st = acquire();
#pragma unroll
      for (int s2 = 0; s2 < 2; ++s2) {
        const int sub = half * 2 + s2;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int row = s2 * 16 + j * 8 + g;          // the B operand's column g
          float d[G][4];
#pragma unroll
          for (int grp = 0; grp < G; ++grp) {
            d[grp][0] = d[grp][1] = d[grp][2] = d[grp][3] = 0.f;
            uint32_t w[BITS == 4 ? 2 : 4];
            if constexpr (BITS == 4) {
              const uint2 v = *(const uint2*)(st + row * GE::ROWB + (((2 * grp + (t >> 1)) ^ swz<CH>(row)) << 4) + (t & 1) * 8);
              w[0] = v.x; w[1] = v.y;
            } else {
              const uint4 v = *(const uint4*)(st + row * GE::ROWB + (((4 * grp + t) ^ swz<CH>(row)) << 4));
              w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w;
            }
#pragma unroll
            for (int step = 0; step < 4; ++step) {
              uint32_t b0, b1;
              if constexpr (BITS == 4) {
                const uint32_t ww = (step & 1) ? w[step >> 1] >> 8 : w[step >> 1];
                b0 = ww & 0x000F000Fu; b1 = ww & 0x00F000F0u;
              } else {
                b0 = w[step] & 0x00FF00FFu; b1 = (w[step] >> 8) & 0x00FF00FFu;
              }
              const uint2 q = qf[grp * 4 + step];
              uint2 ql = make_uint2(0u, 0u);
              if constexpr (QF32) ql = qlo[(grp * 4 + step) * 64];
              mma_f16_16816(d[grp], q.x, ql.x, q.y, ql.y, b0, b1);
            }
          }
          // biases of token g (column g of the tile), scales of this lane's two result columns 2t, 2t + 1
          const int tk = sub * 16 + j * 8;
          float e[4] = {0.f, 0.f, 0.f, 0.f};
          float s0[G], s1[G];
          if constexpr (G == 2) {
            mma_bf16_1688(e, qb, 0u, *(const uint32_t*)(sbb + GE::SB + (tk + g) * 4));
            const uint2 v = *(const uint2*)(sbb + (tk + 2 * t) * 4);
            s0[0] = bf16lo(v.x); s0[1] = bf16hi(v.x); s1[0] = bf16lo(v.y); s1[1] = bf16hi(v.y);
          } else {
            const uint32_t kb = *(const uint16_t*)(sbb + GE::SB + (tk + g) * 2);
            mma_bf16_1688(e, qb, 0u, kb | (kb << 16));
            const uint32_t v = *(const uint32_t*)(sbb + (tk + 2 * t) * 2);
            s0[0] = bf16lo(v); s1[0] = bf16hi(v);
          }
#pragma unroll
          for (int grp = 0; grp < G; ++grp) {
            if constexpr (QF32) { d[grp][0] += d[grp][2]; d[grp][1] += d[grp][3]; }
            e[0] = fmaf(s0[grp], d[grp][0], e[0]);
            e[1] = fmaf(s1[grp], d[grp][1], e[1]);
          }
          sc[sub * 4 + j * 2] = e[0] * C;
          sc[sub * 4 + j * 2 + 1] = e[1] * C;
        }
      }
      __syncwarp();
    }
    if (a.mask) {
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const int tok = tok_blk + (i >> 2) * 16 + ((i >> 1) & 1) * 8 + 2 * t + (i & 1);
        if (tok < n_tok) {
          const int64_t mo = b * a.mask_bstride + t_begin + tok;
          const float mk = a.mask_dtype == QB200_FLOAT32 ? ((const float*)a.mask)[mo] : bf16_bits_to_f32(((const uint16_t*)a.mask)[mo]);
          const float v = fmaf(mk, kLog2e, sc[i]);
          sc[i] = v > kNegBig ? v : kNegBig;
        }
      }
    }
    if (__any_sync(0xffffffffu, tok_blk + kBlk > lim)) {
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const int tok = tok_blk + (i >> 2) * 16 + ((i >> 1) & 1) * 8 + 2 * t + (i & 1);
        if (tok >= lim) sc[i] = kNegBig;
      }
    }
    // ---------------- block softmax bookkeeping ----------------
    // exponent of the block's largest |v_scale|: lanes read the 64 tokens' scales once
    int ex;
    {
      uint32_t m;
      if constexpr (G == 2) {
        const uint2 v = *(const uint2*)(sbb + 2 * GE::SB + lane * 8);
        m = __vmaxu2(v.x & 0x7FFF7FFFu, v.y & 0x7FFF7FFFu);
      } else {
        m = *(const uint32_t*)(sbb + 2 * GE::SB + lane * 4) & 0x7FFF7FFFu;
      }
      ex = (int)(__reduce_max_sync(0xffffffffu, max(m >> 16, m & 0xFFFFu)) >> 7);
    }
    float mb = sc[0];
#pragma unroll
    for (int i = 1; i < 16; ++i) mb = fmaxf(mb, sc[i]);
    mb = fmaxf(mb, __shfl_xor_sync(0xffffffffu, mb, 1));
    mb = fmaxf(mb, __shfl_xor_sync(0xffffffffu, mb, 2));
    // p = 2^(s - r) with r >= max s + ex - 141 keeps p * v_scale below 2^15
    const float r_new = fmaxf(r_run, mb + (float)((ex < 20 ? 20 : ex) - 141));
    if (__any_sync(0xffffffffu, r_new > r_run)) {
      const float alpha = ex2(r_run - r_new);   // 0 while the row was empty
#pragma unroll
      for (int i = 0; i < GE::NT; ++i) { O[i][0] *= alpha; O[i][1] *= alpha; O[i][2] *= alpha; O[i][3] *= alpha; }
#pragma unroll
      for (int i = 0; i < G; ++i) ob[i] *= alpha;
      l_part *= alpha;
      r_run = r_new;
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      sc[i] = sc[i] <= kNegBig ? 0.f : ex2(sc[i] - r_run);
      l_part += sc[i];
    }
    // ---------------- values ----------------
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const uint32_t stv = (uint32_t)__cvta_generic_to_shared(acquire());
#pragma unroll
      for (int s2 = 0; s2 < 2; ++s2) {
        const int sub = half * 2 + s2;
        // A fragments: row g = p * v_scale (hi), row g + 8 = its rest (lo); k slots 2t, 2t + 1 = tokens 2t, 2t + 1,
        // k slots 2t + 8, 2t + 9 = tokens 8 + 2t, 9 + 2t
        uint32_t ah[G][2], al[G][2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int tk = sub * 16 + j * 8 + 2 * t;
          const float p0 = sc[sub * 4 + j * 2], p1 = sc[sub * 4 + j * 2 + 1];
          if constexpr (G == 2) {
            const uint2 v = *(const uint2*)(sbb + 2 * GE::SB + tk * 4), w = *(const uint2*)(sbb + 3 * GE::SB + tk * 4);
            split2(p0 * bf16lo(v.x), p1 * bf16lo(v.y), ah[0][j], al[0][j]);
            split2(p0 * bf16hi(v.x), p1 * bf16hi(v.y), ah[G - 1][j], al[G - 1][j]);
            ob[0] = fmaf(p0, bf16lo(w.x), fmaf(p1, bf16lo(w.y), ob[0]));
            ob[G - 1] = fmaf(p0, bf16hi(w.x), fmaf(p1, bf16hi(w.y), ob[G - 1]));
          } else {
            const uint32_t v = *(const uint32_t*)(sbb + 2 * GE::SB + tk * 2), w = *(const uint32_t*)(sbb + 3 * GE::SB + tk * 2);
            split2(p0 * bf16lo(v), p1 * bf16hi(v), ah[0][j], al[0][j]);
            ob[0] = fmaf(p0, bf16lo(w), fmaf(p1, bf16hi(w), ob[0]));
          }
        }
        // matrix row 4u + i of ldmatrix = token {2u, 8 + 2u, 2u + 1, 9 + 2u}[i]
        const int mr = lane & 15, half_m = lane >> 4;
        const int tokrow = s2 * 16 + 2 * (mr >> 2) + ((mr >> 1) & 1) + 8 * (mr & 1);
#pragma unroll
        for (int kb = 0; kb < CH; kb += 2) {
          uint32_t r[4];
          ldmatrix_b8_trans_x2(r, stv + tokrow * GE::ROWB + (((kb + half_m) ^ swz<CH>(tokrow)) << 4));
#pragma unroll
          for (int m = 0; m < 4; ++m) {   // matrix kb + (m >> 1), byte columns 8 * (m & 1) + g
            if constexpr (BITS == 4) {
              const int grp = (kb + (m >> 1)) >> 1, tile = (kb * 2 + m) * 2;
              const uint32_t hi = r[m] >> 8;
              mma_f16_16816(O[tile], ah[grp][0], al[grp][0], ah[grp][1], al[grp][1], r[m] & 0x000F000Fu, hi & 0x000F000Fu);
              mma_f16_16816(O[tile + 1], ah[grp][0], al[grp][0], ah[grp][1], al[grp][1], r[m] & 0x00F000F0u, hi & 0x00F000F0u);
            } else {
              const int grp = (kb + (m >> 1)) >> 2, tile = kb * 2 + m;
              mma_f16_16816(O[tile], ah[grp][0], al[grp][0], ah[grp][1], al[grp][1], r[m] & 0x00FF00FFu, (r[m] >> 8) & 0x00FF00FFu);
            }
          }
        }
      }
      __syncwarp();
    }
  }
  cp_async_wait<0>();

  // ---- finish the warp: l and the bias dot are partial over the 4 lanes that share a row ----
  l_part += __shfl_xor_sync(0xffffffffu, l_part, 1);
  l_part += __shfl_xor_sync(0xffffffffu, l_part, 2);
#pragma unroll
  for (int grp = 0; grp < G; ++grp) {
    ob[grp] += __shfl_xor_sync(0xffffffffu, ob[grp], 1);
    ob[grp] += __shfl_xor_sync(0xffffffffu, ob[grp], 2);
  }
  __syncthreads();  // every warp is done with its ring
  // merge buffers (reuse the ring): per warp, then of the CTA: r[8], l[8], o[8][D]
  float* wm = (float*)smem;
  float* wl = wm + (kWarps + 1) * kRows;
  float* wo = wl + (kWarps + 1) * kRows;
  if (t == 0) { wm[warp * kRows + g] = r_run; wl[warp * kRows + g] = l_part; }
  float* mine = wo + (size_t)(warp * kRows + g) * D;
#pragma unroll
  for (int tile = 0; tile < GE::NT; tile += (BITS == 4 ? 2 : 1)) {
    constexpr float k24 = 16777216.f, k20 = 1048576.f;   // codes enter as c * 2^-24 (even dims, 8-bit) or 16 c * 2^-24 (odd)
    if constexpr (BITS == 4) {
      const int grp = tile >> 3;   // two tiles hold the even and the odd ones of 16 dims
      float4 v;
      v.x = fmaf(O[tile][0] + O[tile][2], k24, ob[grp]); v.y = fmaf(O[tile + 1][0] + O[tile + 1][2], k20, ob[grp]);
      v.z = fmaf(O[tile][1] + O[tile][3], k24, ob[grp]); v.w = fmaf(O[tile + 1][1] + O[tile + 1][3], k20, ob[grp]);
      *(float4*)(mine + tile * 8 + 4 * t) = v;
    } else {
      const int grp = tile >> 3;
      *(float2*)(mine + tile * 8 + 2 * t) = make_float2(fmaf(O[tile][0] + O[tile][2], k24, ob[grp]), fmaf(O[tile][1] + O[tile][3], k24, ob[grp]));
    }
  }
  __syncthreads();
  const int rows = p.nq - qt * kRows < kRows ? p.nq - qt * kRows : kRows;
  float* cm = wm + kWarps * kRows;
  float* cl = wl + kWarps * kRows;
  float* co = wo + (size_t)kWarps * kRows * D;
  for (int i = tid; i < rows * D; i += kWarps * 32) {
    const int h = i / D, e = i - h * D;
    float M = kNegBig;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) M = fmaxf(M, wm[w * kRows + h]);
    float L = 0.f, Ov = 0.f;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      const float scl = ex2(wm[w * kRows + h] - M);
      L += wl[w * kRows + h] * scl;
      Ov += wo[(size_t)(w * kRows + h) * D + e] * scl;
    }
    if (p.fused) {
      co[i] = Ov;
      if (e == 0) { cm[h] = M; cl[h] = L; }
    } else {
      const int rq = qt * kRows + h, tq = rq / p.gqa, hh = rq - tq * p.gqa;
      const int64_t pi = (((int64_t)b * a.Hq + hk * p.gqa + hh) * a.Tq + tq) * p.nsplit + split;
      p.part_o[pi * D + e] = Ov;
      if (e == 0) { p.part_m[pi] = M * 0.6931471805599453f; p.part_l[pi] = L; }  // natural-log domain for the merge
    }
  }
  if (p.fused) {
    // out = (sum_r o_r w_r) / (sum_r l_r w_r), w_r = 2^(m_r - max m)  (src/transformer.zig:5194-5203), r over the cluster;
    // the cluster spans the grid's x dimension, every CTA of it finishes its share of the outputs
    if (p.nsplit > 1) cluster_sync_all(); else __syncthreads();
    const uint32_t cm_s = (uint32_t)__cvta_generic_to_shared(cm), cl_s = (uint32_t)__cvta_generic_to_shared(cl),
                   co_s = (uint32_t)__cvta_generic_to_shared(co);
    for (int i = split * kWarps * 32 + tid; i < rows * D; i += p.nsplit * kWarps * 32) {
      const int h = i / D, e = i - h * D;
      float M = kNegBig;
      for (int r = 0; r < p.nsplit; ++r) M = fmaxf(M, ld_cluster_f32(map_to_rank(cm_s + 4u * h, (uint32_t)r)));
      float L = 0.f, Ov = 0.f;
      for (int r = 0; r < p.nsplit; ++r) {
        const float wgt = ex2(ld_cluster_f32(map_to_rank(cm_s + 4u * h, (uint32_t)r)) - M);
        L += ld_cluster_f32(map_to_rank(cl_s + 4u * h, (uint32_t)r)) * wgt;
        Ov += ld_cluster_f32(map_to_rank(co_s + 4u * i, (uint32_t)r)) * wgt;
      }
      const float v = Ov * (L > 0.f ? 1.f / L : (L == L ? 0.f : L));
      const int rq = qt * kRows + h, tq = rq / p.gqa, hh = rq - tq * p.gqa;
      const int64_t off = b * a.o_str[0] + (int64_t)(hk * p.gqa + hh) * a.o_str[1] + tq * a.o_tq + e;
      if constexpr (QF32) ((float*)a.out)[off] = v;
      else ((uint16_t*)a.out)[off] = f32_to_bf16_bits(v);
    }
    if (p.nsplit > 1) cluster_sync_all();   // the peers' shared memory stays alive until everybody has read it
  }
}

}  // namespace

bool kv_f16_supported(const KvAttnArgs& a, const KvSeqTable* seqs) {
  if (a.bits != 4 && a.bits != 8) return false;
  if ((a.D != 64 && a.D != 128) || a.Dv != a.D || a.gs != 64) return false;
  const int64_t gqa = a.Hq / a.Hkv;
  if (gqa < 1 || gqa > 8 || a.Tq < 1 || a.Tq > 8) return false;
  if (a.q_dtype != QB200_BFLOAT16 && a.q_dtype != QB200_FLOAT32) return false;
  if (a.Hkv > 8191 || a.B > 65535 || a.T < 1 || a.T > (1 << 30)) return false;
  // 16-byte aligned code rows; scales and biases may lie anywhere
  if (seqs) {
    if (a.B > kMaxSeqPtrs) return false;
    for (int64_t b = 0; b < a.B; ++b) {
      const KvSeq& q = seqs->s[b];
      if (q.T < 1) return false;
      if ((((uintptr_t)q.kq) & 15) || (((uintptr_t)q.vq) & 15)) return false;
      for (int d = 0; d < 2; ++d)
        if (q.kq_str[d] % 4 != 0 || q.vq_str[d] % 4 != 0) return false;
    }
    return true;
  }
  if ((((uintptr_t)a.kq) & 15) || (((uintptr_t)a.vq) & 15)) return false;
  for (int d = 0; d < 3; ++d)
    if (a.kq_str[d] % 4 != 0 || a.vq_str[d] % 4 != 0) return false;
  return true;
}

namespace {
template <int BITS, int D, bool QF32, class TAB>
cudaError_t launch_f16_inst(const F16K& p, const TAB& tab, dim3 grid, cudaStream_t st) {
  constexpr size_t smem = smem_bytes<BITS, D>();
  auto kern = kv_f16_kernel<BITS, D, QF32, TAB>;
  static bool done[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  {
    std::lock_guard<std::mutex> setup_lk(setup_mutex());   // first use on a device, from any thread
    if (dev < 0 || dev >= 64 || !done[dev]) {
      const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e != cudaSuccess) return e;
      note_reader((const void*)kern);
      if (dev >= 0 && dev < 64) done[dev] = true;
    }
  }
  if (p.fused && p.nsplit > 1) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(kWarps * 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)p.nsplit; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return launch_clusters(cfg, kern, p, tab);
  }
  return launch_kernel(kern, grid, dim3(kWarps * 32), smem, st, p, tab);
}
template <int BITS, int D, class TAB>
cudaError_t launch_f16_q(const F16K& p, const TAB& tab, dim3 grid, cudaStream_t st) {
  return p.a.q_dtype == QB200_FLOAT32 ? launch_f16_inst<BITS, D, true, TAB>(p, tab, grid, st) : launch_f16_inst<BITS, D, false, TAB>(p, tab, grid, st);
}
template <class TAB>
cudaError_t launch_f16_tab(const F16K& p, const TAB& tab, dim3 grid, cudaStream_t st) {
  if (p.a.bits == 4) return p.a.D == 64 ? launch_f16_q<4, 64, TAB>(p, tab, grid, st) : launch_f16_q<4, 128, TAB>(p, tab, grid, st);
  return p.a.D == 64 ? launch_f16_q<8, 64, TAB>(p, tab, grid, st) : launch_f16_q<8, 128, TAB>(p, tab, grid, st);
}
}  // namespace

cudaError_t launch_kv_f16(const KvAttnArgs& a, int nsplit, float* pm, float* pl, float* po, cudaStream_t st, const KvSeqTable* seqs, bool fused) {
  F16K p;
  p.a = a; p.nsplit = nsplit; p.gqa = (int)(a.Hq / a.Hkv);
  p.nq = p.gqa * a.Tq;
  p.qtiles = (p.nq + kRows - 1) / kRows;
  p.fused = fused ? 1 : 0;
  p.part_m = pm; p.part_l = pl; p.part_o = po;
  const dim3 grid((unsigned)nsplit, (unsigned)(a.Hkv * p.qtiles), (unsigned)a.B);
  return seqs ? launch_f16_tab(p, *seqs, grid, st) : launch_f16_tab(p, KvNoTable{}, grid, st);
}

}  // namespace qb
