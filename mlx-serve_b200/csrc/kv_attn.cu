// Decode attention read directly from the affine-quantized KV cache.
//
// Semantics: kv_quant.quantAttention with T_q == 1 (mlx-serve
// src/kv_quant.zig:478-687) = softmax(scale * q.K^T + mask) . V over the
// dequantised cache, K/V kept in fp32 as the packed decode kernel does
// (src/transformer.zig:4890-5006), extended to a batch with per-sequence
// lengths (the additive length mask of src/transformer.zig:10216-10249).
// Two phases like the reference kernel: split-KV partials (m, l,
// unnormalised O) then the merge of src/transformer.zig:5194-5203.
#include <math.h>

#include <type_traits>

#include <cstdlib>

#include "kernels.h"

namespace qb {
namespace {

constexpr int kMaxGqa = 8;
constexpr float kNegBig = -1e30f;  // clamp for fully masked blocks (src/transformer.zig:4957-4958)

struct SplitPlan {
  int nsplit;
  int64_t tokens_per_split;  // multiple of 128
};

// Deterministic in (B, Hkv, T): sizes the workspace, and is the plan of the CUDA-core kernel.  It minimises waves of CTAs
// over the GPU x (128-token blocks per warp of 8 + a fixed per-CTA cost of ~0.7 block times), summed over one and two CTAs
// per SM.
__host__ SplitPlan plan_splits(int64_t B, int64_t Hkv, int64_t T) {
  SplitPlan p;
  const int nsm = sm_count();   // CTA slots: one CTA per SM at 8 bits, two at 4 bits
  const int64_t pairs = B * Hkv > 0 ? B * Hkv : 1;
  int64_t max_ns = (T + 255) / 256;  // at least 256 tokens per split
  if (max_ns < 1) max_ns = 1;
  if (max_ns > 1024) max_ns = 1024;
  double best = -1.0;
  int64_t best_ns = 1, best_tps = 128;
  for (int64_t ns = 1; ns <= max_ns; ++ns) {
    int64_t tps = (T + ns - 1) / ns;
    tps = (tps + 127) / 128 * 128;
    if (tps < 128) tps = 128;
    const int64_t ns_eff = (T + tps - 1) / tps > 0 ? (T + tps - 1) / tps : 1;
    const double per_cta = (double)((tps / 128 + 7) / 8) + 0.7;
    double cost = 0.0;
    for (int slots = nsm; slots <= 2 * nsm; slots += nsm) cost += (double)((pairs * ns_eff + slots - 1) / slots) * per_cta;
    if (best < 0.0 || cost < best - 1e-9) { best = cost; best_ns = ns_eff; best_tps = tps; }
  }
  p.nsplit = (int)best_ns;
  p.tokens_per_split = best_tps;
  return p;
}

// Splits of the fp16 tensor-core kernel.  Three CTAs of 4 warps live on an SM; a CTA's warps take the 64-token blocks of its
// split in turn, so a round of a CTA is 256 tokens, and one with fewer blocks than warps counts half for what it lacks.  At head dim 128 and 4 bits a round
// takes 2.4 us in a CTA that has its SM to itself, 3.2 beside a second one and 4.2 among three (0.55 of that at head dim 64, 1.1 at 8 bits); a CTA's start and end
// take 5 us, the merge of a cluster 0.6 and 0.2 for each split.  Beyond 8 splits the partial results go through memory and a merge launch (1.5 us).  The partials have to fit the workspace the caller was told to
// bring, which plan_splits sized.  Within 8 % (geometric mean) of what 28 shapes take at 1 - 20 splits, 4 to 256 pairs of 500 to
// 32768 tokens; the choice is the best of them or within 1 % for all but the longest verify batch (16 x 16 pairs of 32768: 390 us
// against 351) and 500 tokens at head dim 64 (6.5 against 5.9).  2 sequences x 28 heads x 4 verify positions over 4099 tokens:
// 20.5 us at 6 splits, 19.1 at 8.
__host__ int64_t f16_fit(const KvAttnArgs& a) { return (int64_t)(a.workspace_bytes / sizeof(float)) / (a.B * a.Hq * a.Tq * (2 + a.Dv)); }
__host__ int plan_f16(const KvAttnArgs& a, int64_t qtiles, int max_fused) {
  const int64_t pairs = a.B * a.Hkv * qtiles, nsm = sm_count();
  const int64_t fit = f16_fit(a);
  int64_t max_ns = (a.T + 127) / 128;
  if (max_ns > 1024) max_ns = 1024;
  int64_t best = 1;
  double best_cost = -1.0;
  for (int64_t ns = 1; ns <= max_ns && (ns <= max_fused || ns <= fit); ++ns) {
    const int64_t blocks = ((a.T + ns - 1) / ns + 63) / 64, per_sm = (pairs * ns + nsm - 1) / nsm, full = per_sm / 3, rest = per_sm % 3;
    const double rounds = (0.5 * (double)((blocks + 3) / 4) + 0.125 * (double)blocks) * (a.D == 64 ? 0.55 : 1.0) * (a.bits == 8 ? 1.1 : 1.0);
    double cost = (double)full * (4.2 * rounds + 5.0) + (ns > 1 ? 0.6 : 0.0) + 0.2 * (double)(ns < max_fused ? ns : max_fused);
    if (rest) cost += (rest == 1 ? 2.4 : 3.2) * rounds + 5.0;
    if (ns > max_fused) cost += 1.5;
    if (best_cost < 0.0 || cost < best_cost - 1e-9) { best_cost = cost; best = ns; }
  }
  return (int)best;
}

// Splits of the 4-bit integer kernel where they merge inside a cluster (no partials in memory).  A CTA reads a token of one kv head
// in 4 ns alone on its SM and in 7.6 ns beside a second one, plus about 5 us of start and end and 0.8 us of merge per split.  While
// all CTAs are resident the longest sequence decides, in rounds of 512 tokens a CTA; beyond, CTAs follow one another on the places
// that clusters of that size can take.  A last wave that is nearly empty costs less than half a wave, as its CTAs have their SMs to
// themselves (27 x 8 pairs of 20992 tokens: 1.46 waves of two splits take 134 us, 0.73 of one split 164), and about 3 us more the
// emptier it is, which decides short calls (13 x 8 pairs of 4000: two splits 22.5 us, three in 1.12 waves 30.4); lengths that differ
// (`mean`: mean length / T) blur the waves.  Within 8 % (geometric mean over 1 - 8 splits) of what 26 shapes took, 16 to 512 pairs
// of 1024 to 33280 tokens, equal or spread down to a half; its choice is the best of them or within 5 % for all but four (12 %).
// (Counting whole waves for equal lengths chose up to 34 % worse.)
__host__ double cost_clusters(const KvPlaces& places, int64_t pairs, int64_t T, double mean, int cluster, int ns) {
  const double n = (double)pairs * ns, slots = places.n[cluster], up = (double)((T + 512 * ns - 1) / (512 * ns) * 512);
  if (2.0 * n <= 0.97 * slots) return 0.004 * up + 4.5 + 0.8 * ns;   // (with less to spare some CTAs share an SM)
  if (n <= slots) return 0.0076 * up + 5.0 + 0.8 * ns;
  double waves = n / slots;
  const double empty = ceil(waves) - waves;
  if (mean > 0.95) waves = waves + 0.2 > floor(waves) + 0.4 ? waves + 0.2 : floor(waves) + 0.4;
  else waves += 0.35;
  return (0.0076 * mean * (double)T / ns + 5.0) * waves + 3.0 * empty + 0.8 * ns;
}
// `mean` 0: lengths that only the device knows.  The splits are those that lose least over lengths all alike and lengths spread evenly
// down to half of the longest; below 60 us also, at a tenth of the weight, over one long sequence among short ones, which wants many
// (13 x 8 pairs of 4000 tokens, one and two splits: 21.4 and 23.0 us equal, 20.4 and 15.2 one long).  In a longer call where equal
// lengths want fewer splits, few enough for all CTAs to be resident, the kernel takes those when it finds the lengths alike, several
// pairs to a cluster.  (16 x 8 pairs of 32768 tokens: 4 splits take 106 us spread and 137 equal, 2 splits 116 and 131; the kernel
// that chooses 107 and 134.  Where the CTAs are not all resident, several pairs to a cluster lose: 27 x 8 pairs of 20992, two splits
// alone 134 us, in clusters of four 176.)  Finding out costs the start of every CTA a reduction over the lengths, up to 2 us of a
// small call, so it is left out where the model gives it less than 3 %.
__host__ KvSplits plan_clusters(int64_t pairs, int64_t T, double mean) {
  const double m_spread = mean > 0.0 ? mean : 0.75, m_even = mean > 0.0 ? mean : 1.0;
  const KvPlaces places = kv_fast_places();
  const bool choose = mean <= 0.0 && pairs < (1 << 24);   // (the kernel counts pairs in 32 bits)
  double spread[9], even[9], one[9], least_spread = 1e30, least_even = 1e30, least_one = 1e30;
  int ns_even[9], count = 0;
  for (int c = 1; c <= 8 && (c == 1 || T / c >= 256); count = c++) {
    spread[c] = cost_clusters(places, pairs, T, m_spread, c, c);
    even[c] = cost_clusters(places, pairs, T, m_even, c, c);
    one[c] = cost_clusters(places, 1, T, 1.0, c, c);
    ns_even[c] = c;
    if (choose && even[c] >= 60.0) {
      const double enough = 0.97 * even[c];
      for (int ns = 1; ns < c; ++ns) {
        const double cost = c % ns == 0 && pairs * ns <= places.n[c] ? cost_clusters(places, pairs, T, m_even, c, ns) : 1e30;
        if (cost < enough && cost < even[c]) { even[c] = cost; ns_even[c] = ns; }
      }
    }
    least_spread = spread[c] < least_spread ? spread[c] : least_spread;
    least_even = even[c] < least_even ? even[c] : least_even;
    least_one = one[c] < least_one ? one[c] : least_one;
  }
  int best = 1;
  double best_loss = 1e30;
  for (int c = 1; c <= count; ++c) {
    const double loss = spread[c] / least_spread + even[c] / least_even + (mean > 0.0 || least_even >= 60.0 ? 0.0 : 0.1 * one[c] / least_one);
    if (loss < best_loss - 1e-9) { best_loss = loss; best = c; }
  }
  KvSplits s = {best, best, ns_even[best], 0.75f};
  while (s.ns_even != best && s.even_from < 1.f &&
         cost_clusters(places, pairs, T, s.even_from, best, best) < cost_clusters(places, pairs, T, s.even_from, best, s.ns_even))
    s.even_from += 0.03125f;
  return s;
}

struct KvK {
  KvAttnArgs a;
  int nsplit;
  int64_t tps;
  int gqa;
  float* part_m;  // [B, Hq, nsplit]
  float* part_l;  // [B, Hq, nsplit]
  float* part_o;  // [B, Hq, nsplit, Dv]
};

__device__ __forceinline__ float load_mask(const KvK& p, int64_t b, int64_t t) {
  if (!p.a.mask) return 0.f;
  const int64_t off = b * p.a.mask_bstride + t;
  if (p.a.mask_dtype == QB200_FLOAT32) return ((const float*)p.a.mask)[off];
  return bf16_bits_to_f32(((const uint16_t*)p.a.mask)[off]);
}

// Generic CUDA-core path: any head dim that is a multiple of 32, any group
// size, GQA <= 8.  One warp per token; lanes stride over the packed words.
template <int BITS, class TAB>
__global__ void __launch_bounds__(128) kv_split_generic(KvK p, const __grid_constant__ TAB tab) {
  constexpr bool PTRS = std::is_same<TAB, KvSeqTable>::value;
  constexpr int VPW = 32 / BITS;
  extern __shared__ float smem[];
  const KvAttnArgs& a = p.a;
  const int split = blockIdx.x, hk = blockIdx.y;
  const int64_t b = blockIdx.z;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarp = blockDim.x >> 5;
  const int g = p.gqa;
  const int D = (int)a.D, Dv = (int)a.Dv;
  float* qs = smem;                       // [g][D]
  float* red_m = qs + g * D;              // [nwarp][g]
  float* red_l = red_m + nwarp * g;       // [nwarp][g]
  float* red_o = red_l + nwarp * g;       // [nwarp][g][Dv]
  for (int i = threadIdx.x; i < g * D; i += blockDim.x) {
    const int h = i / D, e = i - h * D;
    const int64_t off = b * a.q_str[0] + (int64_t)(hk * g + h) * a.q_str[1] + e;
    qs[i] = a.q_dtype == QB200_FLOAT32 ? ((const float*)a.q)[off] : bf16_bits_to_f32(((const uint16_t*)a.q)[off]);
  }
  __syncthreads();
  // this sequence's cache view: its own pointers and strides, or a slice of the batched tensors
  const uint32_t* kq_b; const uint32_t* vq_b;
  const uint16_t* ks_b; const uint16_t* kb_b; const uint16_t* vs_b; const uint16_t* vb_b;
  int64_t kq_tok, ksb_tok, vq_tok, vsb_tok, T_seq;
  if constexpr (PTRS) {
    const KvSeq& q = tab.s[b];
    kq_b = q.kq + hk * q.kq_str[0]; vq_b = q.vq + hk * q.vq_str[0];
    ks_b = (const uint16_t*)q.ks + hk * q.ksb_str[0]; kb_b = (const uint16_t*)q.kb + hk * q.ksb_str[0];
    vs_b = (const uint16_t*)q.vs + hk * q.vsb_str[0]; vb_b = (const uint16_t*)q.vb + hk * q.vsb_str[0];
    kq_tok = q.kq_str[1]; ksb_tok = q.ksb_str[1]; vq_tok = q.vq_str[1]; vsb_tok = q.vsb_str[1];
    T_seq = q.T;
  } else {
    kq_b = a.kq + b * a.kq_str[0] + hk * a.kq_str[1]; vq_b = a.vq + b * a.vq_str[0] + hk * a.vq_str[1];
    ks_b = (const uint16_t*)a.ks + b * a.ksb_str[0] + hk * a.ksb_str[1]; kb_b = (const uint16_t*)a.kb + b * a.ksb_str[0] + hk * a.ksb_str[1];
    vs_b = (const uint16_t*)a.vs + b * a.vsb_str[0] + hk * a.vsb_str[1]; vb_b = (const uint16_t*)a.vb + b * a.vsb_str[0] + hk * a.vsb_str[1];
    kq_tok = a.kq_str[2]; ksb_tok = a.ksb_str[2]; vq_tok = a.vq_str[2]; vsb_tok = a.vsb_str[2];
    T_seq = a.T;
  }
  int64_t len = a.kv_lens ? (int64_t)a.kv_lens[b] : T_seq;
  if (len > T_seq) len = T_seq;
  const int64_t t0 = (int64_t)split * p.tps;
  int64_t t1 = t0 + p.tps;
  if (t1 > len) t1 = len;

  const int kwords = D / VPW, vwords = Dv / VPW;
  const int vw_per_lane = (vwords + 31) / 32;  // <= 2 for Dv <= 256 at 8 bits
  float m[kMaxGqa], l[kMaxGqa];
  float o[kMaxGqa][2][VPW];
#pragma unroll
  for (int h = 0; h < kMaxGqa; ++h) {
    m[h] = kNegBig; l[h] = 0.f;
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int k = 0; k < VPW; ++k) o[h][j][k] = 0.f;
  }
  for (int64_t t = t0 + warp; t < t1; t += nwarp) {
    const uint32_t* krow = kq_b + t * kq_tok;
    const uint16_t* ksr = ks_b + t * ksb_tok;
    const uint16_t* kbr = kb_b + t * ksb_tok;
    float dot[kMaxGqa];
#pragma unroll
    for (int h = 0; h < kMaxGqa; ++h) dot[h] = 0.f;
    for (int w = lane; w < kwords; w += 32) {
      const uint32_t word = krow[w];
      const int e0 = w * VPW;
      const float sc = bf16_bits_to_f32(ksr[e0 / a.gs]), bi = bf16_bits_to_f32(kbr[e0 / a.gs]);
#pragma unroll
      for (int k = 0; k < VPW; ++k) {
        const float kv = __fadd_rn(__fmul_rn((float)((word >> (k * BITS)) & ((1u << BITS) - 1u)), sc), bi);
#pragma unroll
        for (int h = 0; h < kMaxGqa; ++h)
          if (h < g) dot[h] = fmaf(qs[h * D + e0 + k], kv, dot[h]);
      }
    }
    const float mk = load_mask(p, b, t);
    float pw[kMaxGqa];
#pragma unroll
    for (int h = 0; h < kMaxGqa; ++h) {
      if (h < g) {
        float d = dot[h];
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) d += __shfl_xor_sync(0xffffffffu, d, off);
        float sv = d * a.scale + mk;
        if (!(sv > kNegBig)) sv = kNegBig;  // -inf mask entries and NaN guards
        const float mn = fmaxf(m[h], sv);
        const float alpha = __expf(m[h] - mn);
        pw[h] = sv <= kNegBig ? 0.f : __expf(sv - mn);
        l[h] = l[h] * alpha + pw[h];
        m[h] = mn;
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int k = 0; k < VPW; ++k) o[h][j][k] *= alpha;
      }
    }
    const uint32_t* vrow = vq_b + t * vq_tok;
    const uint16_t* vsr = vs_b + t * vsb_tok;
    const uint16_t* vbr = vb_b + t * vsb_tok;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int w = lane + 32 * j;
      if (j < vw_per_lane && w < vwords) {
        const uint32_t word = vrow[w];
        const int e0 = w * VPW;
        const float sc = bf16_bits_to_f32(vsr[e0 / a.gs]), bi = bf16_bits_to_f32(vbr[e0 / a.gs]);
#pragma unroll
        for (int k = 0; k < VPW; ++k) {
          const float vv = __fadd_rn(__fmul_rn((float)((word >> (k * BITS)) & ((1u << BITS) - 1u)), sc), bi);
#pragma unroll
          for (int h = 0; h < kMaxGqa; ++h)
            if (h < g) o[h][j][k] = fmaf(pw[h], vv, o[h][j][k]);
        }
      }
    }
  }
  // merge the warps of this CTA
  if (lane == 0)
    for (int h = 0; h < g; ++h) { red_m[warp * g + h] = m[h]; red_l[warp * g + h] = l[h]; }
#pragma unroll
  for (int h = 0; h < kMaxGqa; ++h)
    if (h < g)
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int w = lane + 32 * j;
        if (j < vw_per_lane && w < vwords)
#pragma unroll
          for (int k = 0; k < VPW; ++k) red_o[(warp * g + h) * Dv + w * VPW + k] = o[h][j][k];
      }
  __syncthreads();
  for (int i = threadIdx.x; i < g * Dv; i += blockDim.x) {
    const int h = i / Dv, e = i - h * Dv;
    float M = kNegBig;
    for (int w = 0; w < nwarp; ++w) M = fmaxf(M, red_m[w * g + h]);
    float L = 0.f, O = 0.f;
    for (int w = 0; w < nwarp; ++w) {
      const float sc = __expf(red_m[w * g + h] - M);
      L += red_l[w * g + h] * sc;
      O += red_o[(w * g + h) * Dv + e] * sc;
    }
    const int64_t pi = (b * a.Hq + hk * g + h) * p.nsplit + split;
    p.part_o[pi * Dv + e] = O;
    if (e == 0) { p.part_m[pi] = M; p.part_l[pi] = L; }
  }
}

// out = (sum_b o_b w_b) / (sum_b l_b w_b), w_b = exp(m_b - max m)  (src/transformer.zig:5194-5203).  A CTA per output
// row; launched as a programmatic dependent of the split kernel.
__global__ void __launch_bounds__(128) kv_merge(KvK p) {
  const KvAttnArgs& a = p.a;
  __shared__ float wgt[1024];   // plan_splits and plan_f16 cap the splits at 1024
  const int h = blockIdx.x, tq = blockIdx.z;
  const int64_t b = blockIdx.y;
  const int64_t base = ((b * a.Hq + h) * a.Tq + tq) * p.nsplit;
  asm volatile("griddepcontrol.wait;" ::: "memory");
  float M = kNegBig;
  for (int s = threadIdx.x & 31; s < p.nsplit; s += 32) M = fmaxf(M, p.part_m[base + s]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
  float L = 0.f;
  for (int s = threadIdx.x & 31; s < p.nsplit; s += 32) {
    const float w = __expf(p.part_m[base + s] - M);
    if (threadIdx.x < 32) wgt[s] = w;
    L += p.part_l[base + s] * w;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) L += __shfl_xor_sync(0xffffffffu, L, o);
  const float inv = L > 0.f ? 1.f / L : 0.f;
  __syncthreads();
  for (int e = threadIdx.x; e < a.Dv; e += blockDim.x) {
    float O = 0.f;
#pragma unroll 4
    for (int s = 0; s < p.nsplit; ++s) O += p.part_o[(base + s) * a.Dv + e] * wgt[s];
    const int64_t off = b * a.o_str[0] + (int64_t)h * a.o_str[1] + tq * a.o_tq + e;
    const float v = O * inv;
    if (a.q_dtype == QB200_FLOAT32) ((float*)a.out)[off] = v;
    else ((uint16_t*)a.out)[off] = f32_to_bf16_bits(v);
  }
}

}  // namespace

static const Reader kMergeReader((const void*)kv_merge);

cudaError_t launch_kv_fast(const KvAttnArgs& a, KvSplits splits, float* pm, float* pl, float* po, cudaStream_t st, const KvSeqTable* seqs,
                           bool fused);
cudaError_t launch_kv_f16(const KvAttnArgs& a, int nsplit, float* pm, float* pl, float* po, cudaStream_t st, const KvSeqTable* seqs,
                          bool fused);
constexpr int kMaxFusedSplits = 8;   // the portable cluster size

size_t kv_attn_workspace_bytes(int64_t B, int64_t Hq, int64_t Hkv, int64_t T, int64_t Dv) {
  if (B <= 0 || Hq <= 0 || Hkv <= 0 || T <= 0 || Dv <= 0) return 0;
  const SplitPlan sp = plan_splits(B, Hkv, T);
  return (size_t)B * Hq * sp.nsplit * (2 + Dv) * sizeof(float);
}

bool kv_attn_supported(const KvAttnArgs& a) {
  if (a.bits != 4 && a.bits != 8) return false;
  if (a.D % 32 != 0 || a.Dv % 32 != 0) return false;
  if (a.Dv * a.bits / 32 > 64) return false;
  const int64_t gqa = a.Hq / a.Hkv;
  if (gqa < 1 || gqa > kMaxGqa) return false;
  if (a.Hkv > 65535 || a.B > 65535) return false;
  return true;
}

cudaError_t launch_kv_attn(const KvAttnArgs& a, cudaStream_t st, const KvSeqTable* seqs) {
  KvK p;
  p.a = a;
  if (a.B <= 0 || a.Hq <= 0 || a.Hkv <= 0 || a.T <= 0 || a.Dv <= 0 || a.workspace == nullptr) return cudaErrorInvalidValue;
  const SplitPlan sp = plan_splits(a.B, a.Hkv, a.T);
  p.nsplit = sp.nsplit;
  p.tps = sp.tokens_per_split;
  p.gqa = (int)(a.Hq / a.Hkv);
  float* ws = (float*)a.workspace;
  p.part_m = ws;
  p.part_l = ws + a.B * a.Hq * sp.nsplit;
  p.part_o = ws + 2 * a.B * a.Hq * sp.nsplit;
  cudaError_t e;
  if (kv_fast_supported(a, seqs)) {
    // Up to 8 splits per (sequence, kv head) run as one thread-block cluster whose rank 0 merges the partial results
    // through distributed shared memory and writes the output: no partials in global memory, no merge launch.
    // Measured against the merge kernel on one GPU (16 sequences, 8 kv heads): 4-bit caches 23.4 against 24.0 us at
    // 4096 tokens and 132.8 against 134.0 us at 32768; 8-bit caches, whose CTAs fill an SM alone, 33.0 against 31.8 us
    // at 4096 tokens -- so only the 4-bit kernel takes the cluster form.
    if (sp.nsplit <= kMaxFusedSplits && a.bits == 4) {
      double mean = a.kv_lens ? 0.0 : 1.0;
      if (seqs) {
        mean = 0.0;
        for (int64_t b = 0; b < a.B; ++b) mean += (double)seqs->s[b].T / (double)(a.B * a.T);
      }
      e = launch_kv_fast(a, plan_clusters(a.B * a.Hkv, a.T, mean), p.part_m, p.part_l, p.part_o, st, seqs, true);
      if (e == cudaSuccess) return e;
      (void)cudaGetLastError();   // a cluster this launch could not place: fall back to partials and the merge kernel
    }
    e = launch_kv_fast(a, KvSplits{sp.nsplit, sp.nsplit, sp.nsplit, 2.f}, p.part_m, p.part_l, p.part_o, st, seqs, false);
  } else if (kv_f16_supported(a, seqs)) {
    // Head dim 64, GQA 5..8 and the verify widths.  They ran on the CUDA-core kernel before: 2 sequences x 28 query heads x 4
    // verify positions over 4099 tokens at 8 bits 858 -> 20 us, 7 x 14 heads over 22k tokens 1775 -> 38 us, head dim 64
    // 346 -> 10 us.  For GQA <= 4 at head dim 128 the integer kernel above spends fewer instructions per token (two planes
    // of 4 heads fill its MMA columns) and is faster: 133 against 203 us for 16 x 32k tokens.
    // Up to 8 splits per (sequence, kv head, query tile) merge inside a cluster here too, at both code widths.
    p.nsplit = plan_f16(a, (p.gqa * a.Tq + 7) / 8, kMaxFusedSplits);
    if (p.nsplit <= kMaxFusedSplits) {
      e = launch_kv_f16(a, p.nsplit, nullptr, nullptr, nullptr, st, seqs, true);
      if (e == cudaSuccess || p.nsplit == 1) return e;
      (void)cudaGetLastError();   // a cluster this launch could not place: partials and the merge kernel, for as many splits as fit
      if (p.nsplit > f16_fit(a)) p.nsplit = (int)f16_fit(a);
      if (p.nsplit <= 1) return launch_kv_f16(a, 1, nullptr, nullptr, nullptr, st, seqs, true);   // (one split: no cluster)
    }
    const int64_t parts = a.B * a.Hq * a.Tq * p.nsplit;
    p.part_m = ws; p.part_l = ws + parts; p.part_o = ws + 2 * parts;
    e = launch_kv_f16(a, p.nsplit, p.part_m, p.part_l, p.part_o, st, seqs, false);
  } else {
    const int nwarp = 4;
    const size_t smem = (size_t)(p.gqa * a.D + 2 * nwarp * p.gqa + nwarp * p.gqa * a.Dv) * sizeof(float);
    dim3 grid((unsigned)sp.nsplit, (unsigned)a.Hkv, (unsigned)a.B);
    const dim3 blk(nwarp * 32);
    if (seqs) {
      e = a.bits == 4 ? launch_kernel(kv_split_generic<4, KvSeqTable>, grid, blk, smem, st, p, *seqs)
                      : launch_kernel(kv_split_generic<8, KvSeqTable>, grid, blk, smem, st, p, *seqs);
    } else {
      e = a.bits == 4 ? launch_kernel(kv_split_generic<4, KvNoTable>, grid, blk, smem, st, p, KvNoTable{})
                      : launch_kernel(kv_split_generic<8, KvNoTable>, grid, blk, smem, st, p, KvNoTable{});
    }
  }
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)a.Hq, (unsigned)a.B, (unsigned)a.Tq);
  cfg.blockDim = dim3(128);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kv_merge, p);
}

}  // namespace qb
