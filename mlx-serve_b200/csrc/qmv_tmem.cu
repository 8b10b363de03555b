// Quantized matmul for 9 .. 64 tokens with the weights streamed through tensor memory: y[M, N] = x[M, K] . What[N, K]^T, every packed
// word read once, What = bf16(q*s + b) as the dense route that it stands for has it (mlx-serve src/transformer.zig:20987-21011; the
// widths its scheduler batches, src/scheduler.zig:5147, and prompts of a few dozen tokens).
//
// Bound: what a unit of 128 rows x 256 K costs.  At 27 tokens (57344 x 4096, ncu) it takes 770 issue slots of a scheduler over all roles and
// 1359 cycles, with four warps a scheduler to fill them; its 18 KB would take 820 at the copy bandwidth, the tensor pipe is busy for 19 %.
// us a layer of Llama-3-8B's projections (218 M weights, four launches, each replayed), before -> after: 16 tokens
// 85 -> 55, 27 tokens 110 -> 57 (a streaming kernel on mma.sync before), 64 tokens 143 -> 66 (tcgen05 with the weights through shared
// memory); 4096 x 4096 alone 17.2 -> 9.2 at 32, 26.9 -> 10.6 at 64; 512 x 512 8.1 -> 3.5, 7.2 -> 4.1.
//  * A thread converts a weight row.  Its codes lie in a lane of registers and go to the same lane of tensor memory, the A operand of
//    the MMA: no shuffles, no shared-memory tile, scale and bias one register each.
//  * A group of four warps takes units in turn, half a unit (64 columns of tensor memory) at a time, and meets its issuer at a named barrier
//    per slot without waiting; whether the next slot and the next codes are there is looked at while the stores of this half end.  An
//    accumulator per group, as two threads' MMAs into one have no order; the epilogue's warps add them, from the tile's first unit's on.
//  * One thread copies packed codes (128-byte rows), scales and biases by TMA, one x, the B operand as it is.
//  * The CTAs of a cluster split K, each the same part for every tile of 128 rows that the cluster walks, so that its part of x mostly
//    stays in shared memory.  At the end of a tile each hands its fp32 sums to the CTA that owns the tokens (asynchronous remote
//    stores that count at the owner's barrier), which adds them in rank order and stores: no scratch memory, no waiting for whoever
//    is last, and the order of the sum does not depend on timing.
// Not kept: stream-K over all SMs with partial sums in memory (9 us for the last CTA of a tile); one issuer, with or without a scout, for
// all groups (a poll of a barrier costs 107 cycles, half a unit's MMAs 130); MMAs issued by a converting warp (800 cycles a unit that the
// group waits for); scales read by the converting threads, or by cp.async of 8 bytes a row (their latency, 1000 cycles a unit of one warp);
// the conversion unrolled over a unit (14 KB: an eighth of the rate, waiting for instructions); two forms of the kernel for short and long
// launches (a layer, four deep: 359 us against 303 with one -- launches of different kernels refetch their instructions).
// Every mbarrier wait is bounded.  A role whose wait runs out records a code and issues no more copies or MMAs, so that the waits of the
// others run out in turn and nothing is stored; converting warps and issuers still keep every meeting, and tensor memory is freed.  (The
// loops are delicate: a failure word looked at between two polls, or a limit that is no constant, cost 2 - 5 % of a launch.)
#include "stream_ptx.cuh"
#include "tc_ptx.cuh"

namespace qb {
namespace {

constexpr int kMaxMat = 4, kMaxNt = 64, kMaxCluster = 8;
constexpr int CK = 256;                                   // K values of a unit
constexpr int kMaxCodes = 8, kSlots = 6, kMaxX = 16;      // ring depths: packed codes; A operand (half units, of all groups); units of x in shared memory
// Warps: GRP groups of four that convert, four of the epilogue, one each for codes and x, one issuer a group.  (Three groups: 28672 x 4096
// 31.4 us against 26.6 at 27 tokens, for whose three accumulators tensor memory has room once, not twice; the same at 9.)
constexpr int GRP = 2, kOwn = kSlots / GRP;                // slots of a group
constexpr int kEpi0 = 4 * GRP, kCodesWarp = kEpi0 + 4, kXWarp = kCodesWarp + 1, kMmaWarp = kXWarp + 1, kThreads = (kMmaWarp + GRP) * 32;
constexpr uint32_t kSpin = 1u << 22;                      // polls of a bounded wait
constexpr int kBars = 2 * kMaxCodes + kSlots + 2 * kMaxX + 4 + 4;
constexpr size_t kBarBytes = kBars * 8 + 32, kSmem = 225 * 1024;
// One CTA an SM: each allocates all of tensor memory.  Were there room for a second one of the grid (or of another stream's), it would wait
// for the first one's, its peers for its sums, and another cluster's CTAs the other way round.  (At 16 tokens two an SM, the next launch's
// beside this one's, took 51.7 us a layer of Llama-3-8B's projections against 57.5, and had just that fault.)
constexpr size_t kSmemLeast = 116 * 1024;
static_assert(2 * kSmemLeast > 228 * 1024, "two CTAs would fit an SM");
__device__ int g_tmem_error = 0;                          // 0, or the code of a wait that expired

struct TmMaps { CUtensorMap w[kMaxMat], s[kMaxMat], b[kMaxMat]; };
struct TmK {
  const uint16_t* s[kMaxMat]; const uint16_t* b[kMaxMat]; uint16_t* y[kMaxMat];
  int N[kMaxMat];
  int64_t lds[kMaxMat], ldy[kMaxMat];
  int tile0[kMaxMat + 1];
  int nmat, M, nt;           // nt: tokens padded to 16
  int spb, gshift;           // units of K; group size 64 << gshift
  int cluster, cs, dbufs;    // CTAs that split K; depth of the ring of packed codes; accumulators
  int xs, ring;              // units of x in shared memory: all of this CTA's, or a ring of them
  int rx;                    // buffers for the peers' sums: 2, or 1 where a cluster has one tile
  int sb_tma;                // scales and biases by TMA: their rows are 16-byte aligned
  int early;                 // the weights may be read before the previous grid is complete
  uint32_t polls;            // SHORT: of a wait, before it gives up
};

#define QB_SEL4(arr, i) ((i) == 0 ? (arr)[0] : ((i) == 1 ? (arr)[1] : ((i) == 2 ? (arr)[2] : (arr)[3])))
__device__ __forceinline__ int mat_of(const TmK& p, int tile) {
  int mi = 0;
  if (p.nmat > 1 && tile >= p.tile0[1]) mi = 1;
  if (p.nmat > 2 && tile >= p.tile0[2]) mi = 2;
  if (p.nmat > 3 && tile >= p.tile0[3]) mi = 3;
  return mi;
}
__device__ __forceinline__ bool test_cta(uint64_t* bar, uint32_t parity) {
  uint32_t done;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
               : "=r"(done) : "r"(smem_u32(bar)), "r"(parity) : "memory");
  return done != 0;
}
// A whole warp waits.  All lanes poll (107 cycles when the phase is complete; one lane for the others, 134 and a divergent branch).
__device__ __forceinline__ bool warp_wait(uint64_t* bar, uint32_t parity, uint32_t polls) { return __all_sync(0xffffffffu, wait_cta(bar, parity, polls)); }
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void umma_ta(uint32_t d, uint32_t a, uint64_t bd, uint32_t idesc, uint32_t accum) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
               ::"r"(d), "r"(a), "l"(bd), "r"(idesc), "r"(accum) : "memory");
}
__device__ __forceinline__ void commit1(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15};"
      ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
        "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(taddr));
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
__device__ __forceinline__ uint32_t fma2(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t r;
  asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
  return r;
}

// prmt with all four bits of the selectors (__byte_perm takes three of them)
__device__ __forceinline__ uint32_t prmt4(uint32_t a, uint32_t b, uint32_t sel) {
  uint32_t r;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
  return r;
}
// A code as a bf16 by its bits alone: at 4 bits in bits 3 - 6, c * 2^-130, at 8 in bits 0 - 7, c * 2^-133 (the top bit in the exponent
// field, where it counts as much).  The group's multiplier to go with it: s * 2^130 or s * 2^133 in both halves, exact while |s| is below
// the limit that fits_subnormal() tests (0.25, 0.03).
template <int BITS> __device__ __forceinline__ uint32_t scale_up(uint32_t s16) {
  constexpr uint32_t e0 = 127 + 64, e1 = 127 + (BITS == 4 ? 66 : 69);
  const float v = __uint_as_float(s16 << 16) * __uint_as_float(e0 << 23) * __uint_as_float(e1 << 23);
  return __byte_perm(__float_as_uint(v), 0, 0x3232);
}
template <int BITS> __device__ __forceinline__ bool fits_subnormal(uint32_t s16) { return (s16 & 0x7FFFu) < (BITS == 4 ? 0x3E80u : 0x3D00u); }

// bf16(q*s + b) of two codes.  FITS: S = scale_up(s); else S = s in both halves, and the codes become normal numbers first, by two exact
// multiplications.
template <int BITS, bool FITS> __device__ __forceinline__ uint32_t affine2(uint32_t c, uint32_t S, uint32_t b2) {
  if constexpr (!FITS) {
    asm("mul.rn.bf16x2 %0, %0, %1;" : "+r"(c) : "r"(0x7F007F00u));                              // 2^127
    asm("mul.rn.bf16x2 %0, %0, %1;" : "+r"(c) : "r"(BITS == 4 ? 0x41004100u : 0x42804280u));    // 2^3, 2^6
  }
  return fma2(c, S, b2);
}
// 32 codes in order (4 words at 4 bits, 8 at 8) -> 16 columns of tensor memory
template <int BITS, bool FITS> __device__ __forceinline__ void convert32(const uint32_t (&w)[BITS], uint32_t S, uint32_t b2, uint32_t tcol) {
  uint32_t o[16];
  if constexpr (BITS == 4) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint32_t e = (w[i] << 3) & 0x78787878u, f = (w[i] >> 1) & 0x78787878u;   // even, odd codes
      // (a selector with its top bit set gives copies of that byte's top bit: zeros)
      o[4 * i + 0] = affine2<BITS, FITS>(prmt4(e, f, 0xC480), S, b2);
      o[4 * i + 1] = affine2<BITS, FITS>(prmt4(e, f, 0xD591), S, b2);
      o[4 * i + 2] = affine2<BITS, FITS>(prmt4(e, f, 0xE6A2), S, b2);
      o[4 * i + 3] = affine2<BITS, FITS>(prmt4(e, f, 0xF7B3), S, b2);
    }
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      o[2 * i + 0] = affine2<BITS, FITS>(__byte_perm(w[i], 0, 0x4140), S, b2);
      o[2 * i + 1] = affine2<BITS, FITS>(__byte_perm(w[i], 0, 0x4342), S, b2);
    }
  }
  tmem_st16(tcol, o);
}
// 32 codes, `h`-th of the eight such pieces of a row of a unit (128-byte rows, swizzled)
template <int BITS> __device__ __forceinline__ void read32(const unsigned char* row, int r7, int h, uint32_t (&w)[BITS]) {
#pragma unroll
  for (int i = 0; i < BITS / 4; ++i) {
    const int c = BITS == 4 ? h : 2 * (h & 3) + i;           // 16-byte chunk of the row
    const uint4 v = *(const uint4*)(row + (BITS == 8 ? (h >> 2) * (128 * 128) : 0) + ((c ^ r7) << 4));
    w[4 * i] = v.x; w[4 * i + 1] = v.y; w[4 * i + 2] = v.z; w[4 * i + 3] = v.w;
  }
}
// Half a unit of this thread's row: 128 codes to 64 columns of tensor memory, the next codes on their way meanwhile.  A loop and not
// straight-line code: eight warps at eight places of 14 KB of it ran at an eighth of the rate, waiting for instructions.
template <int BITS, bool FITS> __device__ __forceinline__ void convert_half(const unsigned char* row, int r7, int h, uint32_t sv, uint32_t bv, uint32_t tcol) {
  uint32_t w0[BITS], w1[BITS];
  read32<BITS>(row, r7, 4 * h, w0);
#pragma unroll 1
  for (int g = 4 * h; g < 4 * h + 4; g += 2) {
    const uint32_t s2 = __byte_perm(sv, 0, 0x1010), b2 = __byte_perm(bv, 0, 0x1010), S = FITS ? scale_up<BITS>(sv & 0xFFFFu) : s2;
    read32<BITS>(row, r7, g + 1, w1);
    convert32<BITS, FITS>(w0, S, b2, tcol);
    read32<BITS>(row, r7, (g + 2) & 7, w0);
    convert32<BITS, FITS>(w1, S, b2, tcol + 16);
    tcol += 32;
    sv >>= 16;
    bv >>= 16;
  }
}

__device__ __forceinline__ uint32_t map_rank(uint32_t saddr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(rank));
  return r;
}
__device__ __forceinline__ void arrive_remote(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// 16 bytes into a CTA of the cluster, counted at a barrier there
__device__ __forceinline__ void st_async4(uint32_t dst, const uint32_t (&v)[4], uint32_t bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];"
               ::"r"(dst), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_ld4(uint32_t taddr, uint32_t (&r)[4]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(taddr));
}

// SHORT: the launch says how long a wait may be, for tests of waits that run out
template <int BITS, bool SHORT>
__global__ void __launch_bounds__(kThreads, 1) qmv_tmem_kernel(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ TmMaps wm,
                                                               const __grid_constant__ TmK p) {
  extern __shared__ __align__(1024) unsigned char smem[];
  constexpr int kCodes = 128 * CK * BITS / 8;              // packed codes of a unit: 128-byte rows, one box at 4 bits, two at 8
  constexpr int kStage = kCodes + 2 * 2048;                // and blocks of 8 scales and 8 biases of its rows, 16 bytes each
  // (the warp's number from lane 0: what follows from it is then the same in the whole warp to the compiler, too)
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = tid & 31;
  const int CS = p.cs, XS = p.xs, nt = p.nt, C = p.cluster;
  const uint32_t polls = SHORT ? p.polls : kSpin;
  if (smem_u32(smem) & 1023u) {                            // a misaligned window: all CTAs alike leave, behind whatever comes before
    grid_wait();
    if (tid == 0) atomicCAS(&g_tmem_error, 0, 408);
    return;
  }
  unsigned char* codes = smem;                             // [CS][kStage]
  unsigned char* xs = smem + CS * kStage;                  // [XS][4 k-blocks][nt x 128 bytes]
  unsigned char* rx = xs + XS * nt * 512;                  // [p.rx][C ranks][4-token groups that this CTA owns][128 rows][16 bytes]
  const int gpc = C > 1 ? (nt / 4 + C - 1) / C : 0;        // groups of four tokens a CTA owns at most
  const int rx_buf = C * gpc * 2048;
  uint64_t* codes_full = (uint64_t*)(rx + p.rx * rx_buf);
  uint64_t *codes_empty = codes_full + kMaxCodes, *empty = codes_empty + kMaxCodes, *x_full = empty + kSlots, *x_empty = x_full + kMaxX, *d_full = x_empty + kMaxX,
           *d_empty = d_full + 2, *rx_full = d_empty + 2, *rx_free = rx_full + 2;
  uint32_t* tmem_slot = (uint32_t*)(rx_free + 2);
  volatile int& s_fail = *(volatile int*)(tmem_slot + 1);
  const int rank = C > 1 ? (int)cluster_rank_tc() : 0, cl = (int)blockIdx.x / C, ncl = (int)gridDim.x / C;
  const int k0 = p.spb * rank / C, ku = p.spb * (rank + 1) / C - k0;          // this CTA's units of K
  const int ntiles = p.tile0[kMaxMat], tiles = cl < ntiles ? (ntiles - 1 - cl) / ncl + 1 : 0, total = tiles * ku;
  auto failed = [&](int code) { s_fail = code; atomicCAS(&g_tmem_error, 0, code); };
  // The copying warp: codes, scales and biases, unit by unit.  Scales go through shared memory, too, as many units ahead as the codes:
  // read by the converting threads one unit ahead, their latency was half of a unit's time.  One thread and three or four copies a unit
  // where the scales' rows are 16-byte aligned (blocks of 8: the unit's four or two groups are among them); else all lanes copy scales.
  int l_t = -1, l_k = ku, l_st = 0, l_round = 0, l_row = 0, l_mi = 0;         // the unit copied last
  auto next_unit = [&]() {
    if (++l_k >= ku) {
      l_k = 0;
      const int tile = cl + ++l_t * ncl;
      l_mi = mat_of(p, tile);
      l_row = (tile - QB_SEL4(p.tile0, l_mi)) * 128;
    }
  };
  auto copy_codes = [&]() {
    const int k = k0 + l_k;
    uint64_t* bar = &codes_full[l_st];
    const uint32_t dst = smem_u32(codes + l_st * kStage);
    mbar_expect_tx(bar, (uint32_t)(p.sb_tma ? kStage : kCodes));
    tma_load_2d(dst, &wm.w[l_mi], bar, k * (BITS * 8), l_row);
    if constexpr (BITS == 8) tma_load_2d(dst + kCodes / 2, &wm.w[l_mi], bar, k * 64 + 32, l_row);
    if (p.sb_tma) {
      const int e = (k << (2 - p.gshift)) & ~7;
      tma_load_2d(dst + kCodes, &wm.s[l_mi], bar, e, l_row);
      tma_load_2d(dst + kCodes + 2048, &wm.b[l_mi], bar, e, l_row);
    }
  };
  auto copy_scales = [&]() {                               // (all lanes)
    const int e = (k0 + l_k) << (2 - p.gshift), last = QB_SEL4(p.N, l_mi) - 1;
    const int64_t lds = QB_SEL4(p.lds, l_mi);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int n = l_row + r * 32 + lane;
      const int64_t o = (int64_t)(n < last ? n : last) * lds + e;
      const uint32_t sb = smem_u32(codes + l_st * kStage) + kCodes + (uint32_t)((r * 32 + lane) * 16 + (e & 7) * 2);
      if (p.gshift == 0) { cp_async8(sb, QB_SEL4(p.s, l_mi) + o); cp_async8(sb + 2048, QB_SEL4(p.b, l_mi) + o); }
      else { cp_async4(sb, QB_SEL4(p.s, l_mi) + o); cp_async4(sb + 2048, QB_SEL4(p.b, l_mi) + o); }
    }
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&codes_full[l_st])) : "memory");
  };
  // units [from, to): the first CS into empty stages
  auto copy_units = [&](int from, int to) {
    if (p.sb_tma) {
      if (elect_one()) {
        for (int i = from; i < to; ++i) {
          if (l_round > 0 && !wait_cta(&codes_empty[l_st], (uint32_t)(l_round - 1) & 1, polls)) { failed(407); break; }
          if (s_fail) break;
          next_unit();
          copy_codes();
          if (++l_st == CS) { l_st = 0; ++l_round; }
        }
      }
      __syncwarp();
    } else {
      for (int i = from; i < to; ++i) {
        const bool go = l_round == 0 || warp_wait(&codes_empty[l_st], (uint32_t)(l_round - 1) & 1, polls);
        if (!go && lane == 0) failed(407);
        if (!__all_sync(0xffffffffu, go && !s_fail)) break;
        next_unit();
        if (elect_one()) copy_codes();
        __syncwarp();
        copy_scales();
        if (++l_st == CS) { l_st = 0; ++l_round; }
      }
    }
  };

  // Set-up, each role its part: the first copies of codes and scales are under way before the barriers of the other roles exist.
  if (warp == kCodesWarp) {
    if (lane < CS) { mbar_init(&codes_full[lane], p.sb_tma ? 1 : 1 + 32); mbar_init(&codes_empty[lane], 4); }
    if (lane == 0) s_fail = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n\tfence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
    if (!p.early) grid_wait();
    copy_units(0, CS < total ? CS : total);
  } else if (warp == kXWarp) {
    auto init = [&](uint64_t* bar, int n, int count) { if (lane < n) mbar_init(&bar[lane], (uint32_t)count); };
    init(empty, kSlots, 1);
    init(x_full, kMaxX, 1); init(x_empty, kMaxX, 1);
    init(d_full, 2, GRP); init(d_empty, 2, 4);
    init(rx_full, 2, 1); init(rx_free, 2, C > 1 ? 4 * (C - 1) : 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n\tfence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
  }
  __syncthreads();
  if (C > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  // Tensor memory: another launch's CTA may still hold it.  The copying warps need none and go on.
  uint32_t tmem = 0, a0 = 0;
  if (warp != kCodesWarp && warp != kXWarp) {
    if (warp == kEpi0) {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512u));
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    asm volatile("bar.sync 1, %0;" ::"r"(kThreads - 64) : "memory");
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    a0 = tmem + 512 - kSlots * 64;
  }
  auto peers_ready = [&] { if (C > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); };   // once by every thread

  if (warp < kEpi0) {
    // ---- convert this thread's weight row, unit by unit ----
    const int grp = warp >> 2, q = warp & 3, r = q * 32 + lane, mine = total > grp ? (total - grp + GRP - 1) / GRP : 0;
    const uint32_t a_g = a0 + grp * (kOwn * 64) + ((uint32_t)(q * 32) << 16);
    bool ok = true;
    int st = grp, cround = 0, slot = 0, round = 0;           // (CS is a multiple of GRP: a stage is always for the same group)
    int e = (k0 + grp % ku) << (2 - p.gshift), k = grp % ku; // the unit's first group of scales
    uint2 sv, bv;
    auto read_scales = [&]() {
      const unsigned char* sbp = codes + st * kStage + kCodes + r * 16 + (e & 7) * 2;
      if (p.gshift == 0) {
        sv = *(const uint2*)sbp;
        bv = *(const uint2*)(sbp + 2048);
      } else {
        const uint32_t s2 = *(const uint32_t*)sbp, b2 = *(const uint32_t*)(sbp + 2048);
        sv = make_uint2(__byte_perm(s2, 0, 0x1010), __byte_perm(s2, 0, 0x3232));
        bv = make_uint2(__byte_perm(b2, 0, 0x1010), __byte_perm(b2, 0, 0x3232));
      }
    };
    bool codes_ready = false, slot_ready = true;
    int i = 0, h = 0;
    for (; i < mine; ++i) {
      if (!codes_ready) {
        ok = warp_wait(&codes_full[st], (uint32_t)cround & 1, polls);
        read_scales();
      }
      if (!ok) break;
      const unsigned char* row = codes + st * kStage + r * 128;
      uint64_t* done = &codes_empty[st];
      const bool fits = __all_sync(0xffffffffu, fits_subnormal<BITS>(sv.x) && fits_subnormal<BITS>(sv.x >> 16) && fits_subnormal<BITS>(sv.y) && fits_subnormal<BITS>(sv.y >> 16));
#pragma unroll 1
      for (h = 0; h < 2; ++h) {
        if (!slot_ready) ok = warp_wait(&empty[grp * kOwn + slot], (uint32_t)(round - 1) & 1, polls);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t a_s = a_g + (uint32_t)slot * 64;
        if (fits) convert_half<BITS, true>(row, r & 7, h, sv.x, bv.x, a_s);
        else convert_half<BITS, false>(row, r & 7, h, sv.x, bv.x, a_s);
        sv.x = sv.y;
        bv.x = bv.y;
        // what the next half needs is looked for while this one's stores end
        const int id = 2 + grp * kOwn + slot;
        if (++slot == kOwn) { slot = 0; ++round; }
        slot_ready = round == 0 || test_cta(&empty[grp * kOwn + slot], (uint32_t)(round - 1) & 1);
        if (h) {
          st += GRP;
          if (st >= CS) { st -= CS; ++cround; }
          k += GRP;
          while (k >= ku) k -= ku;
          e = (k0 + k) << (2 - p.gshift);
          codes_ready = i + 1 < mine && __all_sync(0xffffffffu, test_cta(&codes_full[st], (uint32_t)cround & 1));
          if (codes_ready) read_scales();
        }
        slot_ready = __all_sync(0xffffffffu, slot_ready);
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        asm volatile("bar.arrive %0, 160;" ::"r"(id) : "memory");
        if (h && lane == 0) mbar_arrive(done);               // (only now that the words have been consumed)
      }
      if (!ok) break;
    }
    if (!ok) {
      // A wait ran out: this warp converts no more, but keeps its meetings with the issuer, each behind the one before in that slot, which
      // the issuer frees whatever happens.  (Met ahead of it, the named barrier would count this warp for the issuer; both would then wait
      // for good.)
      if (lane == 0 && !s_fail) failed(404);
      __syncwarp();
      for (int n = 2 * (mine - i) - (h == 1); n > 0; --n) {
        if (round > 0) warp_wait(&empty[grp * kOwn + slot], (uint32_t)(round - 1) & 1, 8 * kSpin);
        asm volatile("bar.arrive %0, 160;" ::"r"(2 + grp * kOwn + slot) : "memory");
        if (++slot == kOwn) { slot = 0; ++round; }
      }
    }
    __syncwarp();
    peers_ready();
  } else if (warp < kCodesWarp) {
    // ---- epilogue: a thread per weight row, the tokens are the accumulator's columns ----
    const int q = warp & 3, r = q * 32 + lane, ng = nt / 4;
    const int g0 = ng * rank / C, g1 = ng * (rank + 1) / C;                   // groups of four tokens that this CTA stores
    const uint32_t lane_off = (uint32_t)(q * 32) << 16, rx_s = smem_u32(rx);
    if (q == 0) {   // (when tensor memory is this CTA's: a dependent that took it first, and waits for this grid, would never give it back)
      grid_wait();
      asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    }
    bool ok = true, seen = false;
    for (int j = 0; j < tiles && ok; ++j) {
      const int tile = cl + j * ncl, d = p.dbufs == 2 ? j & 1 : 0, b = p.rx == 2 ? j & 1 : 0;
      if (C > 1 && g1 > g0 && tid == kEpi0 * 32) mbar_expect_tx(&rx_full[b], (uint32_t)((C - 1) * (g1 - g0) * 2048));
      ok = warp_wait(&d_full[d], (uint32_t)(p.dbufs == 2 ? j >> 1 : j) & 1, polls) && (C == 1 || j < p.rx || warp_wait(&rx_free[b], (uint32_t)(j / p.rx - 1) & 1, polls)) &&
           __all_sync(0xffffffffu, !s_fail);
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const int mi = mat_of(p, tile), n = (tile - QB_SEL4(p.tile0, mi)) * 128 + r;
      const bool row_ok = n < QB_SEL4(p.N, mi);
      const int64_t ldy = QB_SEL4(p.ldy, mi);
      uint16_t* y = QB_SEL4(p.y, mi) + n;
      const uint32_t acc = tmem + (uint32_t)(GRP * d * nt) + lane_off;       // an accumulator per group
      const int off = (int)((int64_t)j * ku % GRP);                           // the group of the tile's first unit
      if (C > 1 && !seen) { peers_ready(); seen = true; }
      const uint32_t dst = rx_s + (uint32_t)(b * rx_buf + rank * gpc * 2048 + r * 16), bar = smem_u32(&rx_full[b]);
      int to = 0, a = 0, e = ng / C;                                          // the owner of a group: groups [a, e)
#pragma unroll 1
      for (int c = 0; c < nt; c += 32) {
        const bool two = c + 16 < nt;
        uint32_t v[32];
        auto load = [&](int o, int h, uint32_t (&u)[16]) { tmem_ld16(acc + (off + o < GRP ? off + o : off + o - GRP) * nt + c + h * 16, u); };
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t u[GRP][16];
          if (h == 0 || two) {
#pragma unroll
            for (int o = 0; o < GRP; ++o)
              if (o < ku) load(o, h, u[o]);
          }
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            float f = __uint_as_float(u[0][i]);
#pragma unroll
            for (int o = 1; o < GRP; ++o)
              if (o < ku) f += __uint_as_float(u[o][i]);
            v[16 * h + i] = __float_as_uint(f);
          }
        }
        if (c + 32 >= nt) {                                                   // the accumulators may be overwritten
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) mbar_arrive(&d_empty[d]);
        }
        if (C > 1) {
#pragma unroll
          for (int i = 0; i < 8; ++i) {                                       // every group of four tokens to the rank that stores it
            const int g = c / 4 + i;
            if (i >= 4 && !two) break;
            while (g >= e) { ++to; a = e; e = ng * (to + 1) / C; }
            const uint32_t o4[4] = {v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]};
            if (to != rank) st_async4(map_rank(dst + (uint32_t)(g - a) * 2048, (uint32_t)to), o4, map_rank(bar, (uint32_t)to));
            else *(uint4*)(rx + b * rx_buf + (rank * gpc + g - a) * 2048 + r * 16) = make_uint4(o4[0], o4[1], o4[2], o4[3]);
          }
        } else {
          uint16_t* to_y = y + (int64_t)c * ldy;                              // (with a product for every address tiles of few units waited for this: 1.7 us a tile at K = 256 and 512, now 1.3)
          const int left = row_ok ? p.M - c : 0;
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            if (i % 8 == 0 && c + i >= p.M) break;
            if (i < left) *to_y = f32_to_bf16_bits(__uint_as_float(v[i]));
            to_y += ldy;
          }
        }
      }
      if (C > 1 && g1 > g0) {
        ok = warp_wait(&rx_full[b], (uint32_t)(j / p.rx) & 1, polls) && __all_sync(0xffffffffu, !s_fail);
        if (!ok) break;
#pragma unroll 1
        for (int g = g0; g < g1; ++g) {
          const float4* f = (const float4*)(rx + b * rx_buf + (g - g0) * 2048 + r * 16);
          float4 s = f[0];
          for (int o = 1; o < C; ++o) {   // rank order: the sum does not depend on who was ready when
            f += gpc * 128;
            s.x += f->x; s.y += f->y; s.z += f->z; s.w += f->w;
          }
          const float v[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (row_ok && g * 4 + i < p.M) y[(int64_t)(g * 4 + i) * ldy] = f32_to_bf16_bits(v[i]);
        }
        __syncwarp();
      }
      // the peers may send the sums of another tile (for this warp's rows)
      if (C > 1 && j + p.rx < tiles && lane < C && lane != rank) arrive_remote(map_rank(smem_u32(&rx_free[b]), (uint32_t)lane));
    }
    if (!ok && !s_fail) failed(405);
    __syncwarp();
    if (!ok && C > 1 && !seen) peers_ready();
  } else if (warp == kCodesWarp) {
    if (CS < total) copy_units(CS, total);
    __syncwarp();
    peers_ready();
  } else if (warp == kXWarp) {
    if (elect_one()) {
      grid_wait();                                         // x, and whatever used y last
      const uint32_t kb = (uint32_t)nt * 128u;
      auto load_x = [&](int k, int st) {
        mbar_expect_tx(&x_full[st], 4 * kb);
        const uint32_t dst = smem_u32(xs) + (uint32_t)st * 4 * kb;
#pragma unroll
        for (int j = 0; j < 4; ++j) tma_load_2d(dst + j * kb, &xmap, &x_full[st], (k0 + k) * CK + j * 64, 0);
      };
      if (!p.ring) {
        for (int k = 0; k < ku && !s_fail; ++k) load_x(k, k);
      } else {
        int k = 0, st = 0, round = 0;
        for (int i = 0; i < total; ++i) {
          if (round > 0 && !wait_cta(&x_empty[st], (uint32_t)(round - 1) & 1, polls)) { failed(403); break; }
          if (s_fail) break;
          load_x(k, st);
          if (++k == ku) k = 0;
          if (++st == XS) { st = 0; ++round; }
        }
      }
    }
    __syncwarp();
    peers_ready();
  } else {
    // ---- a group's issuer: the MMAs of every half unit that the group has converted, into the group's accumulator ----
    const int grp = warp - kMmaWarp;
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (((uint32_t)nt >> 3) << 17) | ((128u >> 4) << 24);   // f32 += bf16 x bf16, M = 128
    const uint64_t dhi = make_desc(0) & 0xFFFFFFFF00000000ull;
    const uint32_t xd0 = (uint32_t)make_desc(smem_u32(xs)), a_g = a0 + grp * (kOwn * 64), xk = (uint32_t)nt * 8;
    bool ok = true;
    auto wait = [&](uint64_t* bar, int phase) { if (ok) ok = warp_wait(bar, (uint32_t)phase & 1, polls); };
    int slot = 0, xi = grp % XS, xround = 0, k = grp;        // (a ring's XS is a multiple of GRP, too)
    for (int t = 0; t < tiles; ++t, k -= ku) {
      const int d = p.dbufs == 2 ? t & 1 : 0, dround = p.dbufs == 2 ? t >> 1 : t;
      const uint32_t dt = tmem + (uint32_t)((d * GRP + grp) * nt);
      const bool mine = k < ku;
      if (dround > 0) wait(&d_empty[d], dround - 1);
      uint32_t acc = 0;
      if (!p.ring) xi = k;
      for (; k < ku; k += GRP) {
        // (x that stays: units of K change groups from tile to tile where ku is odd, so a group has met all of its units after GRP tiles)
        if (p.ring || t < GRP) wait(&x_full[xi], xround);
#pragma unroll 1
        for (int h = 0; h < 2; ++h) {
          asm volatile("bar.sync %0, 160;" ::"r"(2 + grp * kOwn + slot) : "memory");
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          if (!ok) {                                         // a wait ran out: no more MMAs, but the converting warps go by these meetings
            if (lane == 0) mbar_arrive(&empty[grp * kOwn + slot]);
          } else if (elect_one()) {
            const uint32_t xd = xd0 + (uint32_t)((xi * 4 + h * 2) * nt * 8), a_s = a_g + (uint32_t)slot * 64;
#pragma unroll
            for (int m = 0; m < 8; ++m) umma_ta(dt, a_s + m * 8, dhi | (xd + (m >> 2) * xk + 2 * (m & 3)), idesc, m > 0 ? 1u : acc);
            commit1(smem_u32(&empty[grp * kOwn + slot]));
            if (h > 0 && p.ring) commit1(smem_u32(&x_empty[xi]));
            if (h > 0 && k + GRP >= ku) commit1(smem_u32(&d_full[d]));
          }
          __syncwarp();
          acc = 1;
          if (++slot == kOwn) slot = 0;
        }
        xi += GRP;
        if (p.ring && xi >= XS) { xi -= XS; ++xround; }
      }
      if (!mine && ok && lane == 0) mbar_arrive(&d_full[d]);   // (a tile of fewer units than groups)
      __syncwarp();
    }
    if (!ok && !s_fail) failed(401);
    if (s_fail)
      for (int i = 0; i < 1000; ++i) __nanosleep(1000);    // (MMAs may still be on their way)
    __syncwarp();
    peers_ready();
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == kEpi0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
  // Whatever peers send here has been waited for: every sum, and every arrival that allows another one.  Unless a wait ran out: then
  // copies may still be on their way, and the peers are let go first (a thread that has exited counts as arrived).
  if (s_fail) {
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);
    __syncthreads();
    if (C > 1) cluster_sync_tc();
  }
}

cudaLaunchConfig_t config(cudaLaunchAttribute (&attr)[2], int grid, int cluster, size_t smem, cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = (unsigned)cluster; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  return cfg;
}
// Clusters of this size that the device holds at once (0: none), looked up once per device; index 1: its SMs.
template <int BITS>
cudaError_t clusters_of(int cluster, int* n) {
  static int cached[64][kMaxCluster + 1] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  const int sms = sm_count();
  std::lock_guard<std::mutex> lk(setup_mutex());
  if (cached[dev][0] == 0) {
    auto kern = qmv_tmem_kernel<BITS, false>;
    for (auto k : {kern, qmv_tmem_kernel<BITS, true>}) {
      e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem);
      if (e != cudaSuccess) return e;
      note_reader((const void*)k);
    }
    cached[dev][1] = sms;
    for (int c = 2; c <= kMaxCluster; ++c) {
      cudaLaunchAttribute attr[2];
      cudaLaunchConfig_t cfg = config(attr, sms / c * c, c, kSmem, nullptr);
      cfg.attrs = &attr[1];
      cfg.numAttrs = 1;
      int q = 0;
      if (cudaOccupancyMaxActiveClusters(&q, kern, &cfg) != cudaSuccess) { (void)cudaGetLastError(); q = 0; }
      cached[dev][c] = q < sms / c ? q : sms / c;
    }
    cached[dev][0] = 1;
  }
  *n = cached[dev][cluster];
  return cudaSuccess;
}

// The cluster size: tiles x units of a tile's share, and the hand-over of the sums, which the first tile of a cluster hides better than those
// behind it (its last CTA then waits for the peers' epilogues and the start of its own next tile).  In units of about 0.65 us; by times of
// every size over 1618 shapes (9 - 64 tokens, 1 - 625 tiles, K 256 - 14336).  With 0.4 a tile it took clusters of many short tiles: 4-bit 18945
// x 1280 at 9 tokens, six tiles of one unit a cluster of five, 21.7 us, now two of five units a CTA, 9.8; 28672 x 4096 26.1 -> 22.9.
struct Plan { int cluster, ncl, per, ku; };                // CTAs that split K, clusters, tiles and units of K of one at most
template <int BITS>
cudaError_t plan(const TmK& p, int most, Plan* out) {
  const int ntiles = p.tile0[kMaxMat];
  double best = -1.0;
  for (int c = 1, n = 0; c <= most && c <= p.spb; ++c) {
    const cudaError_t e = clusters_of<BITS>(c, &n);
    if (e != cudaSuccess) return e;
    if (n < 1) continue;
    const int t = (ntiles + n - 1) / n, ku = (p.spb + c - 1) / c;
    const double cost = t * ku + (c > 1 ? 1.4 + 1.6 * (t - 1) : 0.0);
    if (best < 0 || cost < best - 1e-9) { best = cost; *out = {c, n < ntiles ? n : ntiles, t, ku}; }
  }
  return best < 0 ? cudaErrorInvalidConfiguration : cudaSuccess;
}

template <int BITS>
cudaError_t launch_inst(const CUtensorMap& xmap, const TmMaps& wm, TmK p, cudaStream_t st) {
  constexpr int stage = 128 * CK * BITS / 8 + 2 * 2048;
  p.dbufs = 2 * GRP * p.nt <= 128 ? 2 : 1;                 // 512 columns of tensor memory: 6 x 64 for the A operand, groups x accumulators x tokens
  for (int most : {kMaxCluster, 1}) {                      // (where the device places no such cluster: CTAs by themselves)
    Plan pl;
    cudaError_t e = plan<BITS>(p, most, &pl);
    if (e != cudaSuccess) return e;
    const int c = pl.cluster, xu = p.nt * 512, rx1 = c > 1 ? c * ((p.nt / 4 + c - 1) / c) * 2048 : 0, room = (int)(kSmem - kBarBytes);
    p.cluster = c;
    p.rx = pl.per > 1 && c > 1 && room - 2 * rx1 >= 3 * xu + 3 * stage ? 2 : 1;
    const int left = room - p.rx * rx1;
    const int keep = pl.per > 1 ? 4 : 6;                   // x whole where that leaves four stages of codes; six where it is read once
    p.ring = (left - keep * stage) / xu < pl.ku || pl.ku > kMaxX;
    p.xs = pl.ku;
    if (p.ring) {
      p.xs = (left - 6 * stage) / xu;
      p.xs = p.xs > kMaxX ? kMaxX : (p.xs > 3 ? p.xs : 3);
      if (left - p.xs * xu < 3 * stage) p.xs = 2;
      p.xs = p.xs < GRP ? GRP : p.xs / GRP * GRP;
    }
    p.cs = (left - p.xs * xu) / stage;
    if (p.cs > kMaxCodes) p.cs = kMaxCodes;
    p.cs = p.cs / GRP * GRP;
    if (p.cs < GRP) return cudaErrorInvalidConfiguration;
    const size_t smem = (size_t)(p.cs * stage + p.xs * xu + p.rx * rx1) + kBarBytes;
    cudaLaunchAttribute attr[2];
    const cudaLaunchConfig_t cfg = config(attr, pl.ncl * c, c, smem < kSmemLeast ? kSmemLeast : smem, st);
    auto kern = wait_polls() == 0 ? qmv_tmem_kernel<BITS, false> : qmv_tmem_kernel<BITS, true>;
    e = c > 1 ? launch_clusters(cfg, kern, xmap, wm, p) : cudaLaunchKernelEx(&cfg, kern, xmap, wm, p);
    if (e == cudaSuccess || c == 1) return e;
    (void)cudaGetLastError();
  }
  return cudaErrorInvalidConfiguration;
}
}  // namespace

bool qmv_tmem_supported(const QmmArgs& a) {
  if (!a.transpose || a.nbatch != 1 || a.x_dtype != QB200_BFLOAT16) return false;
  if (!((a.bits == 4 || a.bits == 8) && (a.gs == 64 || a.gs == 128))) return false;
  if (a.M <= 8 || a.M > kMaxNt || a.N < 1 || a.N > (1 << 24) || a.K < CK || a.K % CK != 0 || a.K > (1 << 20)) return false;
  if ((((uintptr_t)a.x) & 15) != 0 || (a.ldx * 2) % 16 != 0 || (((uintptr_t)a.w) & 15) != 0 || (a.ldw * 4) % 16 != 0) return false;
  if (a.ldx < a.K || a.ldw * 32 < a.K * a.bits) return false;   // broadcast or overlapping rows: no form of a tensor map
  const uintptr_t al = a.gs == 64 ? 7 : 3;   // a unit's scales in one access
  if ((((uintptr_t)a.s) & al) != 0 || (((uintptr_t)a.b) & al) != 0 || (a.lds * 2) & (int64_t)al) return false;
  return get_encode() != nullptr;
}

// `count` (<= 4) weight matrices on the same activations
cudaError_t launch_qmv_tmem_multi(const QmmArgs* a, int count, cudaStream_t st) {
  TmK p = {};
  TmMaps wm;
  CUtensorMap xmap;
  const int bits = a[0].bits;
  p.nmat = count;
  p.M = (int)a[0].M;
  p.nt = (p.M + 15) & ~15;
  p.spb = (int)(a[0].K / CK);
  p.gshift = a[0].gs == 128 ? 1 : 0;
  int tiles = 0;
  p.sb_tma = 1;
  for (int i = 0; i < kMaxMat; ++i) {
    const QmmArgs& q = a[i < count ? i : 0];
    p.s[i] = (const uint16_t*)q.s + q.sb.offset(0);
    p.b[i] = (const uint16_t*)q.b + q.sb.offset(0);
    p.y[i] = (uint16_t*)q.y + q.yb.offset(0);
    p.N[i] = i < count ? (int)q.N : 0;
    p.lds[i] = q.lds; p.ldy[i] = q.ldy;
    p.tile0[i] = tiles;
    if (i < count) tiles += ((int)q.N + 127) / 128;
    p.sb_tma = p.sb_tma && q.lds % 8 == 0 && q.lds >= q.K / q.gs && (((uintptr_t)p.s[i] | (uintptr_t)p.b[i]) & 15) == 0;
  }
  for (int i = 0; i < count; ++i) {
    const QmmArgs& q = a[i];
    const int64_t groups = q.K / q.gs;
    if (!make_map(&wm.w[i], CU_TENSOR_MAP_DATA_TYPE_UINT32, q.w + q.wb.offset(0), q.K * bits / 32, q.N, q.ldw * 4, 32, 128)) return cudaErrorInvalidValue;
    if (p.sb_tma && (!make_map(&wm.s[i], CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, p.s[i], groups, q.N, q.lds * 2, 8, 128, CU_TENSOR_MAP_SWIZZLE_NONE) ||
                     !make_map(&wm.b[i], CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, p.b[i], groups, q.N, q.lds * 2, 8, 128, CU_TENSOR_MAP_SWIZZLE_NONE)))
      return cudaErrorInvalidValue;
  }
  p.tile0[kMaxMat] = tiles;
  if (!make_map(&xmap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, (const uint16_t*)a[0].x + a[0].xb.offset(0), a[0].K, a[0].M, a[0].ldx * 2, 64, p.nt)) return cudaErrorInvalidValue;
  p.early = weights_settled(st);
  p.polls = wait_polls() > 0 ? (uint32_t)wait_polls() : 0;
  return bits == 8 ? launch_inst<8>(xmap, wm, p, st) : launch_inst<4>(xmap, wm, p, st);
}
cudaError_t launch_qmv_tmem(const QmmArgs& a, cudaStream_t st) { return launch_qmv_tmem_multi(&a, 1, st); }

void qmv_tmem_error_reset() {
  const int zero = 0;
  cudaMemcpyToSymbol(g_tmem_error, &zero, sizeof(int));
}
int qmv_tmem_error_code() {
  int v = 0;
  cudaMemcpyFromSymbol(&v, g_tmem_error, sizeof(int));
  return v;
}

}  // namespace qb
