// Wide prefill on CTA pairs: y[M, N] = x[M, K] . What[N, K]^T with What = bf16(q*s + b), many tokens, dense or grouped (rows
// sorted by expert).  Same definition as the one-CTA kernel in qmm_tc.cu (weight term rounded to bf16 once, fp32 accumulation in
// tensor memory; mlx-serve src/transformer.zig:20987-21011, :15007-15035), which serves what this one declines.
//
// Bound: the tensor core at 512 tokens a tile, the hand-over of a stage between the roles below about 350.  A pair of CTAs
// (tcgen05 cta_group::2) multiplies 256 weight rows by up to 512 tokens: M = 256 rows, 128 of them in either CTA, N = up to 256
// tokens twice, half of them in either CTA.  A CTA so converts 128 x 64 weights and moves about 960 cycles' worth of shared memory
// for 1024 cycles of MMA; one CTA on a 256 x 208 tile, the form before, converted 208 x 64 and moved 1230 for 832.  Weight rows are
// the M side because their number is a multiple of 256 in most models while token counts are ragged: N goes in steps of 32, so an
// expert of 270 rows costs 288 and the tokens of a prompt divide evenly over the waves of tiles.
//
//  * Cluster of two CTAs, persistent, one pair per two SMs.  A tile is one or two units of up to 256 tokens.  Accumulators: a
//    ring of 16 blocks of 32 columns of tensor memory.  A unit takes the next blocks, the epilogue gives every block back as soon as it
//    has read it, and so works beside the next tile except for the blocks that two tiles have in common (two tiles of 288 tokens: 64
//    of 512 columns).  With two slots of 256 columns a tile of two units began after the whole epilogue of the one before, 6800 of
//    16800 cycles at K = 768 (128 experts, us, before -> after: 256 rows an expert 768 x 2048 123 -> 117, 2048 x 768 134 -> 115; 290
//    rows 132 -> 124, 148 -> 126).  Launches of one-unit tiles are a form of their own, without the arithmetic of cut tiles, which take
//    the two halves in turn and give one back at the end of a tile: with one form for both they took 150 cycles a block and 0.2 us a tile more (us, two slots,
//    one form, two forms: 2048 tokens, 14336 x 256 25.6, 29.0, 25.2; 1138 tokens, 14147 x 768 53.3, 59.1, 53.7).
//  * Roles per CTA: twelve warps convert weights (three groups of four that take k-blocks in turn, a thread per weight row), four
//    are the epilogue, and one each loads x, loads packed codes, issues the MMAs (CTA 0 only: its instructions read both CTAs'
//    operands) and scouts for the issuer (CTA 0).  These four share a scheduler without any converting warp: beside one, the
//    issuer took 450 cycles for four MMAs, its few instructions refetched each time.  Copies and converters of CTA 1 arrive at
//    CTA 0's barrier of the stage; one commit frees the stage in both.
//  * What a k-block costs beside its MMAs is synchronisation (measured with the work left out), so: one lane polls for a group of
//    warps and the others follow at a named barrier (polls by all lanes are served one after another and delay the copies'
//    arrivals); no cluster-scope release or acquire on the barriers (each was a fence of about 2000 cycles); the scout runs ahead of
//    the issuer through a named barrier per stage; the issuer's operands are warp-uniform.
// us, before -> after: 2048 tokens, 14336 x 4096 224 -> 162, 4096 x 14336 284 -> 157, 4096 x 4096 98 -> 52, 4096^3 at 8 bits
// 194 -> 95 (1.3 - 1.5 PFLOP/s); 4096 tokens x 8 of 128 experts 768 x 2048 180 -> 125, 2048 x 768 199 -> 137.
// Every mbarrier wait is bounded: on expiry the kernel records a code, the role leaves its loops, tensor memory is freed.
#include "tc_ptx.cuh"

namespace qb {
namespace {

constexpr int BK = 64, RAWB = 2, DQG = 3, WPG = 4, SMAX = 6;
// warps with warp % 4 == 3 share a scheduler, and leave it to the roles that the others wait for
constexpr int kMmaWarp = 3, kScoutWarp = 7, kXWarp = 11, kWWarp = 15, kEpi0 = 16, kThreads = 20 * 32;
constexpr int TILE = 128 * BK * 2, RAW = 128 * 128;   // 128 rows of one k-block as bf16; of one piece of packed codes
constexpr int kMaxE = 256;                            // experts whose tables fit beside the rings; more take the room of a sixth stage
// two units a tile: 4 stages of weights and two boxes of x; one unit: 6 stages of weights and one
constexpr size_t kTiles = (size_t)12 * TILE + RAWB * RAW;
constexpr int kCols = 16;                            // accumulators: a ring of blocks of 32 columns of tensor memory
constexpr int kBars = 2 * SMAX + 2 * RAWB + 2 * kCols;
constexpr size_t smem_of(bool grouped) { return kTiles + kBars * 8 + 48 + (grouped ? 2 * (kMaxE + 1) * 4 : 0); }
static_assert(smem_of(true) <= 227 * 1024, "shared memory");
// Limit of a bounded wait: 2^22 polls, each held by the hardware for kNap ns at most -- a lone waiter's for all of it; in this kernel, where
// other barriers of the CTA change all the time, 360 ns whatever kNap says (20 us to 1 ms: 6300 polls in the 2.3 ms an epilogue waits
// at K = 196608) -- so 1.5 to 8 seconds.  (2^12 polls ended after 1.5 ms, 2^18 after 95 ms, which longer contractions outlive.  A
// limit by the clock, in a function of its own behind 4096 polls, made the roles save registers around the call: 64 experts x 768 x
// 2048 with 5168 rows 52.5 -> 54.0 us.)
constexpr uint32_t kSpin = 1u << 22;

__device__ int g_pair_error = 0;                 // 0, or the code of a wait that expired

struct PairK {
  const uint16_t* s; const uint16_t* b; uint16_t* y;
  int64_t lds, ldy;
  int M, N, K, gshift, sb_vec, y_vec;
  int hmax, stages;                              // tokens per tile at most: 512 (two units, 4 stages) or 256 (one unit, 6; many experts 5)
  int h, tiles_m, ntiles;                        // dense: tokens per tile (multiple of 32)
  const void* rhs; int rhs_i64; int E;           // grouped: expert of every row, ascending
};
struct Tile {
  int row0, row_end, q;                          // tokens [row0, row_end), in steps of 32
  int units, nn0, nn1, col0, col1;               // units of nn0 and nn1 tokens (multiples of 32, up to 256), from these blocks of columns on
  int n0, nend, wrow0, wlast;                    // output columns; first weight row of the tile, last one of the matrix
};
// (a shared::cluster address)
__device__ __forceinline__ void arrive_addr(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void arrive_if(uint32_t bar, bool yes) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %1, 0;\n\t@p mbarrier.arrive.shared::cluster.b64 _, [%0];\n\t}" ::"r"(bar), "r"((uint32_t)yes) : "memory");
}
// A whole warp waits: one lane polls (thirty-two lanes polling one barrier are served one after another, and sixteen warps of them
// kept the copies' own arrivals waiting for thousands of cycles), the others follow.
template <class F>
__device__ __forceinline__ bool warp_wait(int lane, F poll) {
  int ok = 1;
  if (lane == 0) ok = poll();
  return __shfl_sync(0xffffffffu, ok, 0) != 0;
}
// a copy into this CTA whose bytes count at a barrier of either CTA of the pair (a shared::cluster address)
__device__ __forceinline__ void tma_load_pair(uint32_t dst, const CUtensorMap* map, uint32_t bar, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
               ::"r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y) : "memory");
}
// Both by the elected lane.
__device__ __forceinline__ void umma2(uint32_t d, uint64_t ad, uint64_t bd, uint32_t idesc, uint32_t accum) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
               ::"r"(d), "l"(ad), "l"(bd), "r"(idesc), "r"(accum) : "memory");
}
// arrives at the barrier at this offset in both CTAs once the MMAs issued so far are complete
__device__ __forceinline__ void commit2(uint32_t bar) {
  asm volatile(
      "{\n\t.reg .b16 lo, hi;\n\tmov.b32 {lo, hi}, %1;\n\t"
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], lo;\n\t}"
      ::"r"(bar), "r"(3u) : "memory");
}

template <bool GROUPED>
__device__ __forceinline__ Tile tile_at(const PairK& p, const int* s_off, const int* s_tcum, int tile) {
  Tile c;
  int nb;
  if constexpr (GROUPED) {
    int a = 0, b = p.E;   // s_tcum[a] <= tile < s_tcum[b]
    while (b - a > 1) { const int m = (a + b) >> 1; if (s_tcum[m] <= tile) a = m; else b = m; }
    const int local = tile - s_tcum[a], rows = s_off[a + 1] - s_off[a], tm = (rows + p.hmax - 1) / p.hmax;
    const int h = ((rows + tm - 1) / tm + 31) & ~31;      // tiles of like height
    nb = local / tm;
    c.row0 = s_off[a] + (local - nb * tm) * h;
    c.row_end = s_off[a + 1] < c.row0 + h ? s_off[a + 1] : c.row0 + h;
    c.wrow0 = a * p.N + nb * 256;
    c.wlast = a * p.N + p.N - 1;
  } else {
    nb = tile / p.tiles_m;
    c.row0 = (tile - nb * p.tiles_m) * p.h;
    c.row_end = c.row0 + p.h < p.M ? c.row0 + p.h : p.M;
    c.wrow0 = nb * 256;
    c.wlast = p.N - 1;
  }
  c.n0 = nb * 256;
  c.nend = c.n0 + 256 < p.N ? c.n0 + 256 : p.N;
  c.q = c.row_end > c.row0 ? (c.row_end - c.row0 + 31) >> 5 : 1;
  return c;
}
// Where the accumulators of the next tile lie in the ring.  A unit is contiguous.  Tiles of one unit (TWO = false) take its halves in turn,
// each given back whole (a barrier for every block of 32 columns, and room for more than two short tiles, took longer: 129 - 256 tokens at 4
// bits, us, 28672 x 2048 35.5 against 35.1, 14336 x 768 12.4 against 12.2).  Else a tile that the end would cut is cut there into its two units, or, as one unit, moved to block 0 where
// that does not meet the tile before (two tiles of 224 or 256 tokens take turns uncut: cutting them cost 3 %).
struct Ring { int pos = 0, prev = 0; };          // the next free block; the first one of the tile before
template <bool TWO>
__device__ __forceinline__ void place(Tile& c, Ring& r) {
  const int q = c.q;
  int a = q, pos = r.pos;
  if constexpr (!TWO) {
    c.units = 1;
    c.nn0 = q << 5;
    c.nn1 = 0;
    c.col0 = c.col1 = pos;
    r.pos = pos ^ (kCols / 2);
    return;
  }
  if (q > 8 || (pos + q > kCols && q > r.prev)) {
    a = kCols - pos;
    if (pos + q <= kCols || a > 8 || q - a > 8) {
      a = (q + 1) >> 1;
      if (pos + q > kCols && (pos + a > kCols || q - a > pos)) pos = 0;
    }
  } else if (pos + q > kCols) {
    pos = 0;
  }
  const int b = q - a;
  c.units = b ? 2 : 1;
  c.nn0 = a << 5;
  c.nn1 = b << 5;
  c.col0 = r.prev = pos;
  pos += a;
  if (pos + b > kCols) pos = 0;
  c.col1 = pos;
  r.pos = (pos + b) & (kCols - 1);
}

// The issuer's walk, out of line (as part of the big function its loop compiles into something much slower).  Everything the loop
// uses is broadcast from lane 0, so that the compiler knows it to be the same in the whole warp and keeps it in uniform registers.
struct Walk { uint32_t tmem, w_s, x_s, empty_s, acc_s; int tile0, ntiles, tstride, nkb; const int* s_off; const int* s_tcum; };
template <bool GROUPED, bool TWO>
__device__ __noinline__ void issue_walk(const PairK& p, const Walk a) {
  auto U = [](uint32_t v) { return __shfl_sync(0xffffffffu, v, 0); };
  constexpr uint32_t idesc0 = (1u << 4) | (1u << 7) | (1u << 10) | ((256u >> 4) << 24);   // f32 += bf16 x bf16, M = 256
  const uint64_t hi = make_desc(0) & 0xFFFFFFFF00000000ull;
  const uint32_t wd0 = U((uint32_t)make_desc(a.w_s)), xd0 = U((uint32_t)make_desc(a.x_s)), tmem = U(a.tmem), empty_s = U(a.empty_s), acc_s = U(a.acc_s);
  const int nkb = (int)U((uint32_t)a.nkb), S = (int)U((uint32_t)p.stages), ntiles = (int)U((uint32_t)a.ntiles), tstride = (int)U((uint32_t)a.tstride);
  constexpr uint32_t xstep = (TWO ? 2 : 1) * (TILE >> 4);              // a stage of x, in the descriptor's 16-byte units
  uint32_t st = 0;
  Ring ring;
  for (int tile = (int)U((uint32_t)a.tile0); tile < ntiles; tile += tstride) {
    Tile tc = tile_at<GROUPED>(p, a.s_off, a.s_tcum, tile);
    place<TWO>(tc, ring);
    const uint32_t units = U((uint32_t)tc.units), i0 = U(idesc0 | ((uint32_t)(tc.nn0 >> 3) << 17)), i1 = U(idesc0 | ((uint32_t)(tc.nn1 >> 3) << 17));
    const uint32_t c0 = U((uint32_t)tc.col0), c1 = U((uint32_t)tc.col1), d0 = tmem + c0 * 32, d1 = tmem + c1 * 32;
    for (int kb = 0; kb < nkb; ++kb) {
      asm volatile("bar.sync %0, 64;" ::"r"(1 + st) : "memory");   // the scout has seen the stage (and the accumulators' slots) ready
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t wd = wd0 + st * (TILE >> 4), xd = xd0 + st * xstep;
      if (elect_one()) {
#pragma unroll
        for (int k = 0; k < BK / 16; ++k) umma2(d0, hi | (wd + 2 * k), hi | (xd + 2 * k), i0, kb > 0 || k > 0 ? 1u : 0u);
        const bool last = kb + 1 == nkb;
        if (last) commit2(acc_s + c0 * 8u);
        if (TWO && units == 2) {
#pragma unroll
          for (int k = 0; k < BK / 16; ++k) umma2(d1, hi | (wd + 2 * k), hi | (xd + (TILE >> 4) + 2 * k), i1, kb > 0 || k > 0 ? 1u : 0u);
          if (last) commit2(acc_s + c1 * 8u);
        }
        commit2(empty_s + st * 8u);
      }
      __syncwarp();
      st = st + 1 == (uint32_t)S ? 0 : st + 1;
    }
  }
}

// 32 tokens (columns of tensor memory) of this lane's weight row: neighbouring lanes exchange, so that a store covers two rows
__device__ __forceinline__ void store_cols32(uint16_t* y, int64_t ldy, const uint32_t (&v)[32], int tokens, int n, int nend, bool vec, int lane) {
  if (vec) {
    const uint32_t sel = lane & 1 ? 0x3276u : 0x5410u;
    const int ne = n & ~1;
    uint32_t o[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) o[j] = pack2(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1]));
#pragma unroll
    for (int j = 0; j < 16; ++j) o[j] = __byte_perm(o[j], __shfl_xor_sync(0xffffffffu, o[j], 1), sel);   // even lanes: token 2j, odd: 2j + 1
    uint16_t* q = y + (int64_t)(lane & 1) * ldy + ne;
    if (tokens >= 32 && (n | 31) < nend) {   // (the same in the whole warp: its rows are 32 aligned ones)
#pragma unroll
      for (int j = 0; j < 16; ++j) { *(uint32_t*)q = o[j]; q += 2 * ldy; }
    } else {
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        if (2 * j + (lane & 1) < tokens) {
          if (ne + 1 < nend) *(uint32_t*)q = o[j];
          else if (ne < nend) *q = (uint16_t)o[j];
        }
        q += 2 * ldy;
      }
    }
  } else if (n < nend) {
#pragma unroll
    for (int j = 0; j < 32; ++j)
      if (j < tokens) y[(int64_t)j * ldy + n] = f32_to_bf16_bits(__uint_as_float(v[j]));
  }
}

// TWO: tiles of up to two units, 512 tokens
template <int BITS, bool GROUPED, bool TWO>
__global__ void __launch_bounds__(kThreads, 1) qmm_pair_kernel(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap wmap,
                                                               const __grid_constant__ PairK p) {
  extern __shared__ __align__(1024) unsigned char smem[];
  constexpr int KPS = 128 * 8 / (BK * BITS);   // k-blocks per 128-byte piece of packed codes (4 or 2)
  constexpr int xbox = TWO ? 2 : 1;
  const int S = p.stages;
  unsigned char* w_t = smem;                               // [S][128 x 64 bf16]: this CTA's weight rows
  unsigned char* x_t = smem + S * TILE;                    // [S][units][128 x 64 bf16]: its tokens
  unsigned char* raw = smem + 12 * TILE;                   // [RAWB][128 x 128 bytes of codes]
  uint64_t* full = (uint64_t*)(raw + RAWB * RAW);
  uint64_t *empty = full + SMAX, *raw_full = empty + SMAX, *raw_empty = raw_full + RAWB, *acc_full = raw_empty + RAWB, *acc_empty = acc_full + kCols;
  uint32_t* tmem_slot = (uint32_t*)(acc_empty + kCols);
  volatile int& s_fail = *(volatile int*)(tmem_slot + 1);
  volatile int* s_go = (volatile int*)(tmem_slot + 2);     // [DQG][2]
  int* s_off = (int*)(tmem_slot + 2 + 2 * DQG + 2);                      // [E + 1] first row of every expert
  if (GROUPED && p.E > kMaxE) s_off = (int*)(smem + 10 * TILE);
  int* s_tcum = s_off + p.E + 1;                           // [E + 1] prefix of their tile counts
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rank = (int)cluster_rank_tc();
  const int nkb = p.K / BK, tile0 = (int)blockIdx.x >> 1, tstride = (int)gridDim.x >> 1;

  if (warp == 0) {
    auto init = [&](uint64_t* bar, int n, int count) { if (lane < n) mbar_init(&bar[lane], (uint32_t)count); };
    init(full, SMAX, 1 + 2 * WPG); init(empty, SMAX, 1);
    init(raw_full, RAWB, 1); init(raw_empty, RAWB, WPG * KPS + (KPS < DQG ? DQG - KPS : 0));
    init(acc_full, kCols, 1); init(acc_empty, kCols, 8);
    if (lane == 0) {
      s_fail = (smem_u32(smem) & 1023u) ? 308 : 0;         // misaligned window: every role leaves at once
      if (s_fail) atomicCAS(&g_pair_error, 0, 308);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  int ntiles = p.ntiles;
  if constexpr (GROUPED) {
    for (int e = tid; e <= p.E; e += kThreads) {           // rhs is ascending
      int lo = 0, hi = p.M;
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        const long long v = p.rhs_i64 ? ((const long long*)p.rhs)[mid] : (long long)((const int*)p.rhs)[mid];
        if (v < e) lo = mid + 1; else hi = mid;
      }
      s_off[e] = lo;
    }
    __syncthreads();
    if (warp == 0) {
      const int nn = (p.N + 255) / 256;
      int base = 0;
      for (int e0 = 0; e0 < p.E; e0 += 32) {
        const int e = e0 + lane, nt = e < p.E ? (s_off[e + 1] - s_off[e] + p.hmax - 1) / p.hmax * nn : 0;
        int inc = nt;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) { const int o = __shfl_up_sync(0xffffffffu, inc, d); if (lane >= d) inc += o; }
        if (e < p.E) s_tcum[e] = base + inc - nt;
        base += __shfl_sync(0xffffffffu, inc, 31);
      }
      if (lane == 0) s_tcum[p.E] = base;
    }
  }
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512u));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_sync_tc();                                       // the peer's barriers exist
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  if constexpr (GROUPED) ntiles = s_tcum[p.E];
  uint32_t full0;                                          // CTA 0's barriers of the stages
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(full0) : "r"(smem_u32(full)), "r"(0));
  auto at = [&](int tile) { return tile_at<GROUPED>(p, s_off, s_tcum, tile); };
  auto failed = [&](int code) { s_fail = code; atomicCAS(&g_pair_error, 0, code); };

  if (warp == kXWarp) {
    if (elect_one()) {
      int st = 0, round = 0;
      bool ok = true;
      Ring ring;
      for (int tile = tile0; tile < ntiles && ok; tile += tstride) {
        Tile tc = at(tile);
        place<TWO>(tc, ring);
        // boxes of 64 tokens of unit u that CTA r loads
        auto boxes = [&](int r, int u) {
          const int half = (u ? tc.nn1 : tc.nn0) >> 1, t0 = tc.row0 + (u ? tc.nn0 : 0) + r * half;
          return t0 >= tc.row_end || half == 0 ? 0 : (half > 64 && t0 + 64 < tc.row_end ? 2 : 1);
        };
        const int b0 = boxes(rank, 0), b1 = boxes(rank, 1), all = boxes(0, 0) + boxes(0, 1) + boxes(1, 0) + boxes(1, 1);
        const int t0 = tc.row0 + rank * (tc.nn0 >> 1), t1 = tc.row0 + tc.nn0 + rank * (tc.nn1 >> 1);
        for (int kb = 0; kb < nkb; ++kb) {
          if (round > 0 && !wait_cta(&empty[st], (round - 1) & 1, kSpin)) { failed(303); ok = false; break; }
          if (s_fail) { ok = false; break; }
          if (rank == 0) mbar_expect_tx(&full[st], (uint32_t)(all * (TILE / 2)));   // the copies of both CTAs complete at CTA 0's barrier
          const uint32_t dst = smem_u32(x_t + st * xbox * TILE), bar = full0 + (uint32_t)st * 8u;
          if (b0 > 0) tma_load_pair(dst, &xmap, bar, kb * BK, t0);
          if (b0 > 1) tma_load_pair(dst + TILE / 2, &xmap, bar, kb * BK, t0 + 64);
          if (b1 > 0) tma_load_pair(dst + TILE, &xmap, bar, kb * BK, t1);
          if (b1 > 1) tma_load_pair(dst + TILE + TILE / 2, &xmap, bar, kb * BK, t1 + 64);
          if (++st == S) { st = 0; ++round; }
        }
      }
    }
  } else if (warp == kWWarp) {
    if (elect_one()) {
      int sb = 0;
      bool ok = true;
      for (int tile = tile0; tile < ntiles && ok; tile += tstride) {
        const Tile tc = at(tile);
        const int n = tc.wrow0 + rank * 128;
        for (int k = 0; k < nkb / KPS; ++k, ++sb) {
          const int buf = sb % RAWB;
          if (sb >= RAWB && !wait_cta(&raw_empty[buf], ((sb / RAWB) - 1) & 1, kSpin)) { failed(307); ok = false; break; }
          if (s_fail) { ok = false; break; }
          mbar_expect_tx(&raw_full[buf], (uint32_t)RAW);
          tma_load_2d(smem_u32(raw + buf * RAW), &wmap, &raw_full[buf], k * 32, n);
        }
      }
    }
  } else if (warp == kMmaWarp) {
    if (rank == 0) {
      Walk w;
      w.tmem = tmem; w.w_s = smem_u32(w_t); w.x_s = smem_u32(x_t); w.empty_s = smem_u32(empty); w.acc_s = smem_u32(acc_full);
      w.tile0 = tile0; w.ntiles = ntiles; w.tstride = tstride; w.nkb = nkb; w.s_off = s_off; w.s_tcum = s_tcum;
      issue_walk<GROUPED, TWO>(p, w);
    }
  } else if (warp == kScoutWarp) {
    // The same walk as the issuer's, ahead of it: it arrives at a named barrier per stage, where the issuer meets it (a poll of an
    // mbarrier by the issuing thread costs more than the meeting).  When a wait runs out the scout only paces the issuer, which
    // then multiplies stale stages into accumulators nobody trusts (the status word says so).
    if (rank == 0) {
      int st = 0, round = 0, fail = 0;
      Ring ring;
      uint32_t used = 0, par = 0;                        // blocks that had a tile before; how often, modulo 2
      for (int tile = tile0; tile < ntiles; tile += tstride) {
        Tile tc = at(tile);
        place<TWO>(tc, ring);
        uint32_t mine = 1u << tc.col0;
        if constexpr (TWO) {                             // a lane per block
          mine = (((1u << (tc.nn0 >> 5)) - 1) << tc.col0) | (((1u << (tc.nn1 >> 5)) - 1) << tc.col1);
          const bool held = lane < kCols && (mine & used) >> lane & 1;
          if (!fail && !__all_sync(0xffffffffu, !held || wait_cta(&acc_empty[lane], ~(par >> lane) & 1, kSpin))) fail = 306;
        } else if (!fail && (used & mine) && !warp_wait(lane, [&] { return wait_cta(&acc_empty[tc.col0], ~(par >> tc.col0) & 1, kSpin); })) {
          fail = 306;
        }
        used |= mine;
        par ^= mine;
        for (int kb = 0; kb < nkb; ++kb) {
          if (!fail && !warp_wait(lane, [&] { return wait_cta(&full[st], round & 1, kSpin); })) fail = 301;
          if (!fail) asm volatile("bar.arrive %0, 64;" ::"r"(1 + st) : "memory");
          else {
            if (!s_fail && lane == 0) failed(fail);
            __syncwarp();
            asm volatile("bar.sync %0, 64;" ::"r"(1 + st) : "memory");   // (the arrivals before were met: a wait of seconds lies between)
          }
          if (++st == S) { st = 0; ++round; }
        }
      }
    }
  } else if (warp < kEpi0) {
    const int dq = (warp >> 2) * 3 + (warp & 3), grp = dq / WPG, r = (dq % WPG) * 32 + lane;
    const int ntl = ntiles > tile0 ? (ntiles - tile0 + tstride - 1) / tstride : 0, total = ntl * nkb;
    // scales and biases of this thread's row: windows of 8 values (8 << gshift k-blocks), one window ahead
    const int WL = 8 << p.gshift;
    uint4 s_cur = make_uint4(0, 0, 0, 0), b_cur = s_cur, s_nxt = s_cur, b_nxt = s_cur;
    int f_tl = 0, f_kb = 0;
    auto row_ptrs = [&](int tl, const uint16_t*& sp, const uint16_t*& bp) {
      const Tile tc = at(tile0 + tl * tstride);
      int n = tc.wrow0 + rank * 128 + r;
      n = n < tc.wlast ? n : tc.wlast;
      sp = p.s + (int64_t)n * p.lds;
      bp = p.b + (int64_t)n * p.lds;
    };
    const uint16_t *f_sp = nullptr, *f_bp = nullptr, *c_sp = nullptr, *c_bp = nullptr;   // of the window fetched next; of the current tile
    if (ntl > 0) { row_ptrs(0, f_sp, f_bp); c_sp = f_sp; c_bp = f_bp; }
    auto prefetch = [&]() {
      if (f_kb >= nkb) { f_kb = 0; ++f_tl; if (f_tl < ntl) row_ptrs(f_tl, f_sp, f_bp); }
      if (f_tl < ntl) {
        s_nxt = __ldg((const uint4*)(f_sp + (f_kb >> p.gshift)));
        b_nxt = __ldg((const uint4*)(f_bp + (f_kb >> p.gshift)));
      }
      f_kb += WL;
    };
    if (p.sb_vec) prefetch();
    bool ok = true;
    int tl = 0, kb = grp - DQG, st = grp, round = 0, window = -1, turn = 0, seen = 0;     // (three groups, at least four stages)
    for (int it = grp; it < total; it += DQG) {
      kb += DQG;
      if (kb >= nkb) { kb -= nkb; ++tl; if (!p.sb_vec) row_ptrs(tl, c_sp, c_bp); }
      const int sb = it / KPS, kbl = it % KPS, buf = sb % RAWB;   // nkb is a multiple of KPS
      uint32_t sv2, bv2;
      if (p.sb_vec) {
        if (it >> (3 + p.gshift) != window) { window = it >> (3 + p.gshift); s_cur = s_nxt; b_cur = b_nxt; prefetch(); }
        const int e = (kb >> p.gshift) & 7;
        const uint32_t sw = e < 4 ? (e < 2 ? s_cur.x : s_cur.y) : (e < 6 ? s_cur.z : s_cur.w);
        const uint32_t bw = e < 4 ? (e < 2 ? b_cur.x : b_cur.y) : (e < 6 ? b_cur.z : b_cur.w);
        sv2 = (e & 1) ? __byte_perm(sw, sw, 0x3232) : __byte_perm(sw, sw, 0x1010);
        bv2 = (e & 1) ? __byte_perm(bw, bw, 0x3232) : __byte_perm(bw, bw, 0x1010);
      } else {
        const uint32_t sv = __ldg(c_sp + (kb >> p.gshift)), bv = __ldg(c_bp + (kb >> p.gshift));
        sv2 = sv | (sv << 16);
        bv2 = bv | (bv << 16);
      }
      // one lane of the group polls for the codes and for the stage, the group follows at a named barrier
      if (dq % WPG == 0 && lane == 0) {
        // Pieces without a k-block of this group are seen and released too: a parity names a phase only to who follows every one.
        bool go = true;
        for (; KPS < DQG && seen < sb; ++seen) {
          go = go && wait_cta(&raw_full[seen % RAWB], (seen / RAWB) & 1, kSpin);
          mbar_arrive(&raw_empty[seen % RAWB]);
        }
        seen = sb + 1;
        go = go && wait_cta(&raw_full[buf], (sb / RAWB) & 1, kSpin);
        if (go && round > 0) go = wait_cta(&empty[st], (round - 1) & 1, kSpin);
        s_go[grp * 2 + turn] = go && !s_fail;
      }
      asm volatile("bar.sync %0, 128;" ::"r"(1 + SMAX + grp) : "memory");
      ok = s_go[grp * 2 + turn] != 0;   // (two slots in turn: the next write comes after everybody's read)
      if (!ok) break;
      constexpr int WPH = 32 * BITS / 32;
      uint32_t c[2][WPH];
      const unsigned char* rr = raw + buf * RAW + r * 128;
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int i = 0; i < WPH / 4; ++i) {
          const int chunk = kbl * (WPH / 2) + h * (WPH / 4) + i;
          const uint4 v = *(const uint4*)(rr + ((chunk ^ (r & 7)) << 4));
          c[h][4 * i] = v.x; c[h][4 * i + 1] = v.y; c[h][4 * i + 2] = v.z; c[h][4 * i + 3] = v.w;
        }
      dequant_half<BITS>(c[0], sv2, bv2, w_t + st * TILE, r, 0);
      dequant_half<BITS>(c[1], sv2, bv2, w_t + st * TILE, r, 1);
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) {
        arrive_addr(full0 + (uint32_t)st * 8u);
        mbar_arrive(&raw_empty[buf]);   // (only now that the words have been consumed)
      }
      turn ^= 1;
      st += DQG;
      if (st >= S) { st -= S; ++round; }
    }
    if (!ok && !s_fail) failed(304);
  } else {
    // epilogue: this CTA's 128 weight rows (lanes) x the tokens (columns) of every unit
    const int q = warp & 3;
    Ring ring;
    uint32_t par = 0;                                      // how often a unit began at a block, modulo 2
    bool ok = true;
    for (int tile = tile0; tile < ntiles && ok; tile += tstride) {
      Tile tc = at(tile);
      place<TWO>(tc, ring);
      const int n = tc.n0 + rank * 128 + q * 32 + lane;
      for (int j = 0; j < tc.units; ++j) {
        const int col = j ? tc.col1 : tc.col0;
        ok = warp_wait(lane, [&] { return wait_cta(&acc_full[col], (par >> col) & 1, kSpin); });
        if (!ok || s_fail) { ok = false; break; }
        par ^= 1u << col;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const int t0 = tc.row0 + (j ? tc.nn0 : 0), nt = j ? tc.nn1 : tc.nn0;
        const uint32_t freed = full0 + (uint32_t)((unsigned char*)&acc_empty[col] - (unsigned char*)full);
        const uint32_t acc = tmem + ((uint32_t)(q * 32) << 16) + col * 32;
        if constexpr (TWO) {
          if (n - lane < tc.nend) {   // (a branch around the stores inside the loop, or around the arrival: 150 cycles more a block)
#pragma unroll 1
            for (int c0 = 0; c0 < nt; c0 += 32) {
              uint32_t v[32];
              tmem_ld32(acc + c0, v);
              asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
              asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
              arrive_if(freed + (uint32_t)c0 / 4, lane == 0);    // the block may be overwritten
              store_cols32(p.y + (int64_t)(t0 + c0) * p.ldy, p.ldy, v, tc.row_end - (t0 + c0), n, tc.nend, p.y_vec != 0, lane);
            }
          } else {
            arrive_if(freed + 8 * (uint32_t)lane, lane < nt >> 5);
          }
        } else {               // short enough that the next tile but one does not wait for blocks: given back at the end
          if (n - lane < tc.nend) {
#pragma unroll 1
            for (int c0 = 0; c0 < nt; c0 += 32) {
              uint32_t v[32];
              tmem_ld32(acc + c0, v);
              asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
              store_cols32(p.y + (int64_t)(t0 + c0) * p.ldy, p.ldy, v, tc.row_end - (t0 + c0), n, tc.nend, p.y_vec != 0, lane);
            }
          }
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) arrive_addr(freed);
        }
      }
    }
    if (!ok && !s_fail) failed(305);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_sync_tc();                                       // nobody reads or arrives at the peer's shared memory any more
  if (warp == kMmaWarp) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
}

template <int BITS, bool GROUPED, bool TWO>
cudaError_t launch_inst(const CUtensorMap& xmap, const CUtensorMap& wmap, const PairK& p, int pairs, cudaStream_t st) {
  auto kern = qmm_pair_kernel<BITS, GROUPED, TWO>;
  static bool done[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  {
    std::lock_guard<std::mutex> lk(setup_mutex());   // first use on a device, from any thread
    if (dev < 0 || dev >= 64 || !done[dev]) {
      const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_of(GROUPED));
      if (e != cudaSuccess) return e;
      if (dev >= 0 && dev < 64) done[dev] = true;
    }
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(2 * pairs));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem_of(GROUPED);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return launch_clusters(cfg, kern, xmap, wmap, p);
}
// wrows: weight rows in all (E * N in the grouped form)
cudaError_t launch_pair(PairK& p, const void* x, int64_t ldx, const uint32_t* w, int64_t wrows, int64_t ldw, int bits, bool grouped, int pairs, cudaStream_t st) {
  CUtensorMap xmap, wmap;
  if (!make_map(&xmap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, x, p.K, p.M, ldx * 2, BK, 64)) return cudaErrorInvalidValue;
  if (!make_map(&wmap, CU_TENSOR_MAP_DATA_TYPE_UINT32, w, (int64_t)p.K * bits / 32, wrows, ldw * 4, 32, 128)) return cudaErrorInvalidValue;
  p.sb_vec = p.K % (512 << p.gshift) == 0 && p.lds % 8 == 0 && ((((uintptr_t)p.s) | ((uintptr_t)p.b)) & 15) == 0;
  p.y_vec = p.ldy % 2 == 0 && ((uintptr_t)p.y & 3) == 0;
  p.stages = p.hmax == 512 ? 4 : (grouped && p.E > kMaxE ? 5 : 6);
  const auto launch = p.hmax == 512 ? (grouped ? (bits == 4 ? launch_inst<4, true, true> : launch_inst<8, true, true>)
                                               : (bits == 4 ? launch_inst<4, false, true> : launch_inst<8, false, true>))
                                    : (grouped ? (bits == 4 ? launch_inst<4, true, false> : launch_inst<8, true, false>)
                                               : (bits == 4 ? launch_inst<4, false, false> : launch_inst<8, false, false>));
  return launch(xmap, wmap, p, pairs, st);
}

}  // namespace

// Formats and alignment are those of the one-CTA kernel.  That one remains the faster up to 128 tokens (half tiles, K split over a
// cluster) and, up to 256, for few or long rows (256 tokens, us, pair / one CTA: 14336 x 4096 39 / 52, 6144 x 2048 25 / 37,
// 4096 x 4096 37 / 38, 1024 x 4096 37 / 30, 4096 x 14336 111 / 79), and from 257 below two blocks of rows (300 tokens: 512 x 4096
// 40 / 45).
bool qmm_pair_supported(const QmmArgs& a) {
  return qmm_tc_supported(a) && ((a.M > 256 && a.N >= 512) || (a.M > 128 && a.N >= 6144 && a.K <= a.N));
}
cudaError_t launch_qmm_pair(const QmmArgs& a, cudaStream_t st) {
  PairK p = {};
  p.s = (const uint16_t*)a.s + a.sb.offset(0); p.b = (const uint16_t*)a.b + a.sb.offset(0); p.y = (uint16_t*)a.y + a.yb.offset(0);
  p.lds = a.lds; p.ldy = a.ldy; p.M = (int)a.M; p.N = (int)a.N; p.K = (int)a.K; p.gshift = a.gs == 128 ? 1 : 0;
  const int pairs = sm_count() / 2;
  const int64_t nb = (a.N + 255) / 256;
  // Waves x time of a tile, in us: its k-blocks, and what of the epilogue the next tile's do not hide -- more of it in two units where K is
  // short, and where the rows of y are off 4 bytes and stored value by value.  Fitted to 48 shapes (300 to 4096 tokens, K 2048 to 14336,
  // every height from 96): the height taken is 0.3 % slower than the best of a shape on average, 3.5 % at worst.  Below K = 2048 and for odd
  // rows (74 shapes) 1.1 % and 9.5 %.
  const bool y_vec = p.ldy % 2 == 0 && ((uintptr_t)p.y & 3) == 0;
  const int nkb = p.K / BK;
  double best = -1.0;
  for (int h = 512; h >= 128; h -= 32) {
    const int64_t tiles = ((a.M + h - 1) / h) * nb;
    const double kb = 0.375 + h * 0.00016 + (h > 352 ? (h - 352) * 0.00067 : 0.0);
    const double epi = 1.25 + (h > 256 ? (h - 256) * 0.0207 + 7.0 / nkb : 0.0) + (y_vec ? 0.0 : h / 32 * (h > 256 ? 1.05 : 0.7));
    const double cost = (double)((tiles + pairs - 1) / pairs) * (nkb * kb + epi);
    if (best < 0 || cost < best - 1e-9) { best = cost; p.h = h; }
  }
  p.hmax = p.h > 256 ? 512 : 256;
  p.tiles_m = (int)((a.M + p.h - 1) / p.h);
  p.ntiles = p.tiles_m * (int)nb;
  return launch_pair(p, (const char*)a.x + a.xb.offset(0) * 2, a.ldx, a.w + a.wb.offset(0), a.N, a.ldw, a.bits, false, p.ntiles < pairs ? p.ntiles : pairs, st);
}

// Any number of rows per expert for which a grouped product is the form at all (64 rows, 128 experts of 768 x 2048: 104 us against
// 122 on single CTAs).
bool gather_pair_supported(const GatherArgs& a) { return gather_tc_supported(a) && a.N >= 256; }
cudaError_t launch_gather_pair(const GatherArgs& a, cudaStream_t st) {
  PairK p = {};
  p.s = (const uint16_t*)a.s; p.b = (const uint16_t*)a.b; p.y = (uint16_t*)a.y;
  p.lds = a.K / a.gs; p.ldy = a.N; p.M = (int)a.I; p.N = (int)a.N; p.K = (int)a.K; p.gshift = a.gs == 128 ? 1 : 0;
  p.rhs = a.rhs; p.rhs_i64 = a.rhs_dtype == QB200_INT64; p.E = (int)a.E;
  // two units where many experts have more than 256 rows (128 experts +- 12 %, 768 x 2048 / 2048 x 768, us, two units and one: 256 rows
  // on average 116 / 135 and 115 / 149, 230 113 / 109 and 112 / 115, 180 108 / 106 and 107 / 111)
  p.hmax = a.I > 200 * a.E && a.E <= kMaxE ? 512 : 256;
  return launch_pair(p, a.x, a.K, a.w, a.E * a.N, a.K * a.bits / 32, a.bits, true, sm_count() / 2, st);
}

void qmm_pair_error_reset() {
  const int zero = 0;
  cudaMemcpyToSymbol(g_pair_error, &zero, sizeof(int));
}
int qmm_pair_error_code() {
  int v = 0;
  cudaMemcpyFromSymbol(&v, g_pair_error, sizeof(int));
  return v;
}

}  // namespace qb
