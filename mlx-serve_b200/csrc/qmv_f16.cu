// Weight-streaming quantized matmul for decode and small-batch widths on the fp16 tensor cores:
// y[M, N] = x[M, K] . What[N, K]^T, 4- or 8-bit affine codes, group size 32 / 64 / 128, K any multiple of the group size,
// up to 32 activation columns per launch (bf16: a column per token; fp32: two, high and low part).
//
// Replaces mlx_quantized_matmul(transpose=true) as called by qmatmulBits (mlx-serve src/transformer.zig:20894-20983) at
// decode widths, the small-M verify lanes (src/transformer.zig:1317-1453) and continuous batches.
//
// HBM-bound by its bytes; what such a kernel runs out of before is issue slots, so it spends few of them per code:
//  * A code c in the low bits of a 16-bit half IS the fp16 subnormal c * 2^-24, exactly: an AND turns a packed word into an
//    MMA operand register of two codes.  The nibble above it is 16 c * 2^-24; the activation it meets carries the 1/16.
//    4 bits: four ANDs and one shift per 8 codes.  The weight term is never rounded: sums of code * activation are scaled
//    by the group's scale in fp32, and the bias term is an MMA of its own (biases against the activations' group sums in
//    three bf16 parts).
//  * Activations become fp16 under one power-of-two scale per token and CTA (largest |x| to the top of the range): bf16
//    values within 2^-24 of the token's largest keep all their bits, fp32 ones are split into two columns (22 bits).
//  * Four producer warps stream W rows and the scales and biases (cp.async in 16-byte pieces, those of the scales from the
//    aligned address below: their rows may start anywhere) into a ring of stages; 16 consumer warps split a stage by (group of 64 k) x (16-row tile) and keep their sums in registers over the whole of K, so nothing
//    is reduced until a block of 64 rows is finished, and a group's activation fragments are loaded once for all its tiles.
//  * The CTAs of a cluster split K over the same rows when the activations are many (they would not fit, and every CTA
//    would convert all of them); partial sums meet through distributed shared memory, each CTA finishing its share.
//  * Rows are dealt to the clusters evenly, to the row, across all matrices of the call: no last wave.
//  * Programmatic dependent launch; where the host knows that the kernels before write no weights (weights_settled), the ring fills
//    with them before the wait.
// Measured: 5 tokens x 7211 x 2880 (4-bit) 59 us on the CUDA-core kernel before, see the dispatch rule in api.cu.  The rows
// of a 64-row block end in a sum over eight warps (and the cluster) that stops the consumers, which is what keeps it behind
// the ring-per-warp kernel of qmv_stream.cu at the widths both serve.
#include <type_traits>

#include "kernels.h"
#include "stream_ptx.cuh"

namespace qb {
namespace {

constexpr int kCW = 16;                    // consumer warps
constexpr int kPW = 4;                     // producer warps
constexpr int kThreads = (kCW + kPW) * 32;
constexpr int kKC = 512;                   // K values per stage
constexpr int kGC = kKC / 64;              // 64-wide groups per stage
constexpr int kRB = 64;                    // rows per block
constexpr int kWK = kGC;                   // consumer warps over a stage's groups
constexpr int kWR = kCW / kWK;             // ... times tiles of 16 rows side by side
constexpr int kTPW = kRB / 16 / kWR;       // tiles per warp
constexpr int kSBP = 48;                   // bytes per row of the scale (or bias) window of a stage
constexpr int kMaxMat = 4;

template <int BITS> struct Geo {
  static constexpr int ROWB = kKC * BITS / 8;       // code bytes of a row in a stage
  static constexpr int GB = 64 * BITS / 8;          // ... of a group
  static constexpr int PITCH = ROWB + GB;           // keeps the fragment reads free of bank conflicts
  static constexpr int W = kRB * PITCH;
  static constexpr int STAGE = W + 2 * kRB * kSBP;
};

__device__ int g_f16_error = 0;            // 0, or the code of a bounded wait that expired

struct F16K {
  const void* x;
  const uint32_t* w[kMaxMat]; const uint16_t* s[kMaxMat]; const uint16_t* b[kMaxMat]; void* y[kMaxMat];
  int N[kMaxMat];
  int row0[kMaxMat + 1];   // first row of each matrix in the launch-wide row numbering
  int64_t ldw[kMaxMat], lds[kMaxMat], ldy[kMaxMat];
  int nmat;
  int M, K, x_f32;
  int64_t ldx;
  int cluster;             // CTAs that split K
  int gc;                  // 64-groups per CTA (the last may have fewer)
  int ct;                  // activation columns stored per n8 tile (1, 2, 4, 8)
  int stages;
  int early;               // the weights may be read before the previous grid is complete
  int polls;               // of a wait, before it gives up
};

#define QB_SEL4(arr, i) ((i) == 0 ? (arr)[0] : ((i) == 1 ? (arr)[1] : ((i) == 2 ? (arr)[2] : (arr)[3])))

// Counts this thread's outstanding cp.async copies: one of the barrier's arrivals happens when they have landed.
__device__ __forceinline__ void mbar_arrive_cp_async(uint32_t bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
}
template <bool CLUSTER>
__device__ __forceinline__ bool mbar_poll(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  if constexpr (CLUSTER)
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2, %3;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(bar), "r"(parity), "r"(2000u) : "memory");
  else
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(bar), "r"(parity), "r"(2000u) : "memory");
  return ok != 0;
}
// Bounded: a wait gives up after the polls that the word `polls` in shared memory allows (the hardware holds one for 0.4 to 2 us, so the
// default is a second or more), records `code` if it is the launch's first, and leaves 0 in the word: no wait of the CTA is long after
// that.  The producers then leave their loops, and the consumers leave theirs together at the end of the block of rows, storing
// nothing of it.  (A word and no register: the wider instantiations have none to spare.)
constexpr int kPolls = 1 << 21;
template <bool CLUSTER = false>
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, uint32_t polls, int code) {
  if (mbar_poll<CLUSTER>(bar, parity)) return true;
  int n;
  asm volatile("ld.volatile.shared.u32 %0, [%1];" : "=r"(n) : "r"(polls) : "memory");
  for (; n > 0; --n)
    if (mbar_poll<CLUSTER>(bar, parity)) return true;
  atomicCAS(&g_f16_error, 0, code);
  asm volatile("st.volatile.shared.u32 [%0], %1;" ::"r"(polls), "r"(0u) : "memory");
  return false;
}
__device__ __forceinline__ void consumers_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kCW * 32) : "memory"); }
__device__ __forceinline__ uint32_t lds_u16(uint32_t a) {
  uint16_t v;
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ uint32_t lds_u32(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ uint2 lds_u64(uint32_t a) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a));
  return v;
}
__device__ __forceinline__ uint4 lds_u128(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
  return v;
}

// A block of rows of one matrix: at most kRB rows of this cluster's share.
struct Block { int mi, row, n; };
// The cluster's share [v0, v1) of the launch-wide rows, block by block.
__device__ __forceinline__ bool next_block(const F16K& p, int& v, int v1, Block& b) {
  if (v >= v1) return false;
  b.mi = 0;
  if (p.nmat > 1 && v >= p.row0[1]) b.mi = 1;
  if (p.nmat > 2 && v >= p.row0[2]) b.mi = 2;
  if (p.nmat > 3 && v >= p.row0[3]) b.mi = 3;
  const int r0 = QB_SEL4(p.row0, b.mi);
  int end = r0 + QB_SEL4(p.N, b.mi);
  end = end < v1 ? end : v1;
  b.row = v - r0;
  b.n = end - v < kRB ? end - v : kRB;
  v += b.n;
  return true;
}

// NT: n8 tiles of activation columns; GS: group size
template <int BITS, int NT, int GS>
__global__ void __launch_bounds__(kThreads, 1) qmv_f16_kernel(const __grid_constant__ F16K p) {
  using GE = Geo<BITS>;
  constexpr int SUBS = GS == 32 ? 2 : 1;            // 8-group steps of the bias product per stage
  constexpr int CB = kKC / GS * 2;                  // bytes of scales a row advances per stage
  extern __shared__ __align__(128) unsigned char smem[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int NS = p.stages, cs = p.cluster;
  const int crank = cs > 1 ? (int)cluster_rank() : 0;
  const int nclus = (int)gridDim.x / cs, clus = (int)blockIdx.x / cs;
  const int total = p.row0[p.nmat];
  const int v0 = (int)((int64_t)total * clus / nclus), v1 = (int)((int64_t)total * (clus + 1) / nclus);
  const int k0 = crank * p.gc * 64;                                     // first K value of this CTA
  const int klen = p.K - k0 < p.gc * 64 ? (p.K - k0 > 0 ? p.K - k0 : 0) : p.gc * 64;
  const int nch = (klen + kKC - 1) / kKC;                               // stages per block of rows

  // ---- shared memory ----
  const uint32_t ring = smem_u32(smem);
  unsigned char* sp = smem + (size_t)NS * GE::STAGE;
  unsigned char* xf = sp;  sp += (size_t)p.gc * 2 * NT * p.ct * 64;     // activation fragments [group][word][tile][column, t]
  unsigned char* xb = sp;  sp += (size_t)((p.gc + kGC - 1) / kGC) * SUBS * 3 * NT * 128;   // group sums [step][part][tile][column][8]
  float* recv = (float*)sp; sp += cs > 1 ? (size_t)2 * NT * 2048 : 0;   // partial sums from the cluster [2][rank][tile][512 / cs]
  uint32_t* s_max = (uint32_t*)sp; sp += 32 * 4;
  float* s_ts = (float*)sp; sp += 8 * NT * 4;
  const uint32_t full = smem_u32(sp), empty = full + 8 * NS, rx = empty + 8 * NS;
  const uint32_t polls = rx + 16;                                       // what is left of a wait: 0 once one has run out
  volatile int* pw = (volatile int*)(sp + 16 * NS + 16);                // (that word), and [2]: the consumers leave, by block in turn
  if (tid == 0) {
    pw[0] = p.polls;
    pw[1] = pw[2] = 0;
    for (int i = 0; i < NS; ++i) { mbar_init(full + 8 * i, kPW * 32); mbar_init(empty + 8 * i, kCW); }
    mbar_init(rx, kCW * cs);
    mbar_init(rx + 8, kCW * cs);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (tid < 32) s_max[tid] = 0u;
  __syncthreads();
  if (cs > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");   // waited for before the first remote write

  if (warp >= kCW) {
    // =========================== producer warps: a quarter of a stage's rows each ===========================
    // the kernel before may have written the weights, unless the host knows better
    if (!p.early) asm volatile("griddepcontrol.wait;" ::: "memory");
    constexpr int LPR = GE::ROWB / 16, RPI = 32 / LPR, HR = kRB / kPW;   // lanes per row, rows per copy instruction, rows per warp
    const int r0 = (warp - kCW) * HR, lr = r0 + lane / LPR, lc = (lane % LPR) * 16;
    int v = v0;
    uint32_t st = 0, ph = 1;    // stage index; parity of the wait for its previous readers (the first round passes at once)
    auto advance = [&]() { if (++st == (uint32_t)NS) { st = 0; ph ^= 1; } };
    bool ok = true;
    Block b;
    while (ok && next_block(p, v, v1, b)) {
      const int64_t ldw = QB_SEL4(p.ldw, b.mi) * 4, lds = QB_SEL4(p.lds, b.mi) * 2;
      const unsigned char* wsrc = (const unsigned char*)QB_SEL4(p.w, b.mi) + (size_t)k0 * BITS / 8 + (int64_t)(b.row + lr) * ldw + lc;
      const unsigned char* sbase = (const unsigned char*)QB_SEL4(p.s, b.mi);
      const unsigned char* bbase = (const unsigned char*)QB_SEL4(p.b, b.mi);
      const int64_t slen = (int64_t)(QB_SEL4(p.N, b.mi) - 1) * lds + (int64_t)(p.K / GS) * 2;   // bytes of scales from the base
      int64_t soff = (int64_t)(b.row + r0 + lane) * lds + (int64_t)(k0 / GS) * 2;               // of this lane's row
      const int n = b.n;
      for (int ch = 0; ch < nch; ++ch) {
        ok = mbar_wait(empty + 8 * st, ph, polls, 1);
        if (!ok) break;
        const uint32_t dst = ring + st * GE::STAGE, fb = full + 8 * st;
        const int left = klen - ch * kKC;
        if (lc < left * BITS / 8) {
          const uint32_t d = dst + lr * GE::PITCH + lc;
          const unsigned char* q = wsrc;
#pragma unroll
          for (int i = 0; i < HR / RPI; ++i) {
            if (lr + i * RPI < n) cp_async16(d + i * RPI * GE::PITCH, q);
            q += RPI * ldw;
          }
        }
        wsrc += GE::ROWB;
        if (lane < HR && r0 + lane < n) {
          const int64_t a0 = soff & ~(int64_t)15;
          const uint32_t sd = dst + GE::W + (r0 + lane) * kSBP;
#pragma unroll
          for (int i = 0; i < (CB + 14 + 15) / 16; ++i) {
            const int64_t a = a0 + i * 16, rest = slen - a;
            if (a < soff + CB && rest > 0) {
              const uint32_t nb = rest < 16 ? (uint32_t)rest : 16u;
              cp_async16_z(sd + i * 16, sbase + a, nb);
              cp_async16_z(sd + kRB * kSBP + i * 16, bbase + a, nb);
            }
          }
        }
        soff += CB;
        mbar_arrive_cp_async(fb);
        advance();
      }
      // one stage slot per block is the consumers' scratch for the sums over their K shares
      ok = ok && mbar_wait(empty + 8 * st, ph, polls, 2);
      if (!ok) break;
      mbar_arrive(full + 8 * st);
      advance();
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncwarp();
    if (cs > 1) {
      asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
      cluster_sync_all();   // nobody's shared memory goes away while a peer may still write to it
    }
    return;
  }

  // =========================== consumer warps ===========================
  for (int i = tid; i < ((p.gc + kGC - 1) / kGC) * SUBS * 3 * NT * 32; i += kCW * 32) ((uint32_t*)xb)[i] = 0u;
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

  // ---- stage the activations: one thread per 8 consecutive values of a token ----
  {
    constexpr int PF = NT == 1 ? 4 : (NT == 2 ? 8 : 12);   // items a thread keeps in registers between the two passes
    const int cpt = (klen + 63) / 64 * 8;                  // items per token (whole 64-groups; values behind K are 0)
    const int items = p.M * cpt;
    const bool al16 = ((((uintptr_t)p.x) | (uintptr_t)(p.ldx * (p.x_f32 ? 4 : 2)) | (uintptr_t)(k0 * 2)) & 15) == 0;
    auto run = [&](auto f32tag) {
      constexpr bool F32 = decltype(f32tag)::value;
      constexpr int RW = F32 ? 2 : 1;
      auto load = [&](int i, uint4 (&r)[RW]) {
        const int m = i / cpt, c = i - m * cpt;
#pragma unroll
        for (int j = 0; j < RW; ++j) r[j] = make_uint4(0u, 0u, 0u, 0u);
        if (i >= items || c * 8 >= klen) return;
        const int64_t off = (int64_t)m * p.ldx + k0 + c * 8;
        if constexpr (!F32) {
          const uint16_t* px = (const uint16_t*)p.x + off;
          if (al16) { r[0] = *(const uint4*)px; }
          else {
            uint32_t q[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) q[j] = (uint32_t)px[2 * j] | ((uint32_t)px[2 * j + 1] << 16);
            r[0] = make_uint4(q[0], q[1], q[2], q[3]);
          }
        } else {
          const float* px = (const float*)p.x + off;
          if (al16) { r[0] = *(const uint4*)px; r[RW - 1] = *(const uint4*)(px + 4); }
          else {
            r[0] = make_uint4(__float_as_uint(px[0]), __float_as_uint(px[1]), __float_as_uint(px[2]), __float_as_uint(px[3]));
            r[RW - 1] = make_uint4(__float_as_uint(px[4]), __float_as_uint(px[5]), __float_as_uint(px[6]), __float_as_uint(px[7]));
          }
        }
      };
      auto amax = [&](const uint4 (&r)[RW]) -> uint32_t {   // bit pattern of the largest |x| (fp32), NaN above infinity
        if constexpr (!F32) {
          const uint32_t a = __vmaxu2(__vmaxu2(r[0].x & 0x7FFF7FFFu, r[0].y & 0x7FFF7FFFu), __vmaxu2(r[0].z & 0x7FFF7FFFu, r[0].w & 0x7FFF7FFFu));
          return max(a & 0xFFFF0000u, a << 16);
        } else {
          const uint4 q = r[RW - 1];
          const uint32_t k = 0x7FFFFFFFu;
          return max(max(max(r[0].x & k, r[0].y & k), max(r[0].z & k, r[0].w & k)), max(max(q.x & k, q.y & k), max(q.z & k, q.w & k)));
        }
      };
      uint4 raw[PF][RW];
      const int nq = (items + kCW * 32 - 1) / (kCW * 32);
      auto note = [&](int i, const uint4 (&r)[RW]) {
        uint32_t mx = amax(r);
        mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
        mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
        mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, 4));
        if ((lane & 7) == 0 && i < items) atomicMax(&s_max[i / cpt], mx);
      };
#pragma unroll
      for (int q = 0; q < PF; ++q)
        if (q < nq) load(q * kCW * 32 + tid, raw[q]);
#pragma unroll
      for (int q = 0; q < PF; ++q)
        if (q < nq) note(q * kCW * 32 + tid, raw[q]);
      for (int q = PF; q < nq; ++q) {
        uint4 r[RW];
        load(q * kCW * 32 + tid, r);
        note(q * kCW * 32 + tid, r);
      }
      consumers_sync();
      auto put = [&](int i, const uint4 (&r)[RW]) {
        const bool ok = i < items;
        const int m = ok ? i / cpt : 0, c = i - m * cpt;
        const uint32_t mb = s_max[m];
        int e = (int)(mb >> 23) - 127;                     // |x| < 2^(e + 1)
        e = e < -100 ? -100 : (e > 110 ? 110 : e);
        const float up = pow2i(14 - e);
        float f[8];
        if constexpr (!F32) {
          f[0] = bf16lo(r[0].x); f[1] = bf16hi(r[0].x); f[2] = bf16lo(r[0].y); f[3] = bf16hi(r[0].y);
          f[4] = bf16lo(r[0].z); f[5] = bf16hi(r[0].z); f[6] = bf16lo(r[0].w); f[7] = bf16hi(r[0].w);
        } else {
          const uint4 q = r[RW - 1];
          f[0] = __uint_as_float(r[0].x); f[1] = __uint_as_float(r[0].y); f[2] = __uint_as_float(r[0].z); f[3] = __uint_as_float(r[0].w);
          f[4] = __uint_as_float(q.x); f[5] = __uint_as_float(q.y); f[6] = __uint_as_float(q.z); f[7] = __uint_as_float(q.w);
        }
        float sum = 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) { f[j] *= up; sum += f[j]; }
        sum += __shfl_xor_sync(0xffffffffu, sum, 1);
        sum += __shfl_xor_sync(0xffffffffu, sum, 2);
        if constexpr (GS != 32) sum += __shfl_xor_sync(0xffffffffu, sum, 4);
        if (!ok) return;
        const int gi = c >> 3, cc = c & 7;
        const int tt = GS == 32 ? (cc & 3) : (cc >> 1), jw = GS == 32 ? (cc >> 2) : (cc & 1);
        const int col = F32 ? 2 * m : m, nt = col >> 3, cl = col & 7;
        if ((cc & (GS == 32 ? 3 : 7)) == 0) {
          // column `col` of the bias product: group sums * 2^-24 in three bf16 parts
          const int sg = GS == 32 ? gi * 2 + jw : gi;      // index among groups (of 64, or 32)
          uint16_t* d = (uint16_t*)(xb + (size_t)(sg >> 3) * 3 * NT * 128 + nt * 128 + cl * 16) + (sg & 7);
          float v = sum * 5.9604644775390625e-8f;
#pragma unroll
          for (int k = 0; k < 3; ++k) { const uint16_t h = f32_to_bf16_bits(v); d[k * NT * 64] = h; v -= bf16_bits_to_f32(h); }
        }
        float a[8];   // operand order: (b0, b1) of the word's two MMA steps, pairs
        if constexpr (BITS == 4) {
          a[0] = f[0]; a[1] = f[4]; a[2] = f[1] * 0.0625f; a[3] = f[5] * 0.0625f;
          a[4] = f[2]; a[5] = f[6]; a[6] = f[3] * 0.0625f; a[7] = f[7] * 0.0625f;
        } else {
          a[0] = f[0]; a[1] = f[2]; a[2] = f[1]; a[3] = f[3];
          a[4] = f[4]; a[5] = f[6]; a[6] = f[5]; a[7] = f[7];
        }
        unsigned char* d = xf + ((size_t)(gi * 2 + jw) * NT + nt) * (p.ct * 64) + (cl * 4 + tt) * 16;
        if constexpr (!F32) {
          *(uint4*)d = make_uint4(pack_f16x2(a[0], a[1]), pack_f16x2(a[2], a[3]), pack_f16x2(a[4], a[5]), pack_f16x2(a[6], a[7]));
        } else {
          uint32_t hi[4], lo[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const float h0 = __uint_as_float(__float_as_uint(a[2 * k]) & 0xFFFFE000u), h1 = __uint_as_float(__float_as_uint(a[2 * k + 1]) & 0xFFFFE000u);
            hi[k] = pack_f16x2(h0, h1);
            lo[k] = pack_f16x2(a[2 * k] - h0, a[2 * k + 1] - h1);
          }
          *(uint4*)d = make_uint4(hi[0], hi[1], hi[2], hi[3]);
          *(uint4*)(d + 64) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
        }
      };
#pragma unroll
      for (int q = 0; q < PF; ++q)
        if (q < nq) put(q * kCW * 32 + tid, raw[q]);
      for (int q = PF; q < nq; ++q) {
        uint4 r[RW];
        load(q * kCW * 32 + tid, r);
        put(q * kCW * 32 + tid, r);
      }
      if (tid < 8 * NT) {                                  // factor of a column's sums
        const int m = F32 ? tid >> 1 : tid;
        const uint32_t mb = m < p.M ? s_max[m] : 0u;
        int e = (int)(mb >> 23) - 127;
        e = e < -100 ? -100 : (e > 110 ? 110 : e);
        s_ts[tid] = (mb >> 23) >= 255u ? __uint_as_float(0x7FC00000u) : pow2i(10 + e);
      }
    };
    if (p.x_f32) run(std::true_type{}); else run(std::false_type{});
  }
  consumers_sync();

  const int wk = warp % kWK, wr = warp / kWK;
  const int ngr = (klen + 63) / 64;                                   // 64-groups of this CTA
  const uint32_t xf_s = smem_u32(xf), xb_s = smem_u32(xb);
  const uint32_t xstep = (uint32_t)(NT * p.ct * 64);                  // bytes between the two words of a group
  const uint32_t xlane = xf_s + (uint32_t)(((g & (p.ct - 1)) * 4 + t) * 16) + (uint32_t)wk * 2u * xstep;
  // fragment addresses inside a stage: row g of tile wr, this warp's group, this lane's codes
  const uint32_t wlane = (uint32_t)((wr * 16 + g) * GE::PITCH + wk * GE::GB) + (GS == 32 ? (BITS == 4 ? 4 : 8) * t : (BITS == 4 ? 8 : 16) * t);
  uint32_t st = 0, ph = 0;
  auto advance = [&]() { if (++st == (uint32_t)NS) { st = 0; ph ^= 1; } };
  int v = v0, rxn = 0;                                                // (rxn: blocks finished)
  Block b;
  while (next_block(p, v, v1, b)) {
    float acc[kTPW][NT][4];
#pragma unroll
    for (int tp = 0; tp < kTPW; ++tp)
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) acc[tp][nt][0] = acc[tp][nt][1] = acc[tp][nt][2] = acc[tp][nt][3] = 0.f;
    // scales of row g start this many bytes into the 16-byte window of the first stage (the same for rows g + 8 k)
    const uint32_t sh0 = (uint32_t)((((int64_t)(b.row + g) * QB_SEL4(p.lds, b.mi) + k0 / GS) * 2) & 15);
    for (int ch = 0; ch < nch; ++ch) {
      mbar_wait(full + 8 * st, ph, polls, 3);
      const uint32_t sb = ring + st * GE::STAGE;
      const uint32_t sh = CB % 16 == 0 ? sh0 : ((sh0 + (uint32_t)(ch * CB)) & 15u);
      const uint32_t sa = sb + GE::W + (uint32_t)((wr * 16 + g) * kSBP) + sh;
      if (ch * kGC + wk < ngr) {
        uint4 bf[NT][2];
        const uint32_t xa = xlane + (uint32_t)(ch * kGC) * 2u * xstep;
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
          bf[nt][0] = lds_u128(xa + (uint32_t)(nt * p.ct * 64));
          bf[nt][1] = lds_u128(xa + xstep + (uint32_t)(nt * p.ct * 64));
        }
#pragma unroll
        for (int tp = 0; tp < kTPW; ++tp) {
          if ((tp * kWR + wr) * 16 < b.n) {
            constexpr uint32_t TS = kWR * 16 * GE::PITCH;
            const uint32_t wa = sb + wlane + tp * TS;
            const uint32_t ss = sa + tp * (kWR * 16 * kSBP) + (GS == 64 ? 2 * wk : (GS == 128 ? 2 * (wk >> 1) : 4 * wk));
            uint32_t wl[BITS / 2], wh[BITS / 2];      // packed words of rows g and g + 8
            if constexpr (BITS == 4 && GS != 32) {
              const uint2 a = lds_u64(wa), c = lds_u64(wa + 8 * GE::PITCH);
              wl[0] = a.x; wl[1] = a.y; wh[0] = c.x; wh[1] = c.y;
            } else if constexpr (BITS == 4) {
              wl[0] = lds_u32(wa); wl[1] = lds_u32(wa + 16); wh[0] = lds_u32(wa + 8 * GE::PITCH); wh[1] = lds_u32(wa + 8 * GE::PITCH + 16);
            } else if constexpr (GS != 32) {
              const uint4 a = lds_u128(wa), c = lds_u128(wa + 8 * GE::PITCH);
              wl[0] = a.x; wl[1] = a.y; wl[2] = a.z; wl[3] = a.w; wh[0] = c.x; wh[1] = c.y; wh[2] = c.z; wh[3] = c.w;
            } else {
              const uint2 a = lds_u64(wa), a2 = lds_u64(wa + 32), c = lds_u64(wa + 8 * GE::PITCH), c2 = lds_u64(wa + 8 * GE::PITCH + 32);
              wl[0] = a.x; wl[1] = a.y; wl[2] = a2.x; wl[3] = a2.y; wh[0] = c.x; wh[1] = c.y; wh[2] = c2.x; wh[3] = c2.y;
            }
            float s_lo[GS == 32 ? 2 : 1], s_hi[GS == 32 ? 2 : 1];
#pragma unroll
            for (int h = 0; h < (GS == 32 ? 2 : 1); ++h) {
              s_lo[h] = __uint_as_float(lds_u16(ss + 2 * h) << 16);
              s_hi[h] = __uint_as_float(lds_u16(ss + 8 * kSBP + 2 * h) << 16);
            }
            // A operands of the group's four k16 steps
            uint32_t a0[4], a1[4], a2[4], a3[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              if constexpr (BITS == 4) {
                const uint32_t l = (k & 1) ? wl[k >> 1] >> 8 : wl[k >> 1], h = (k & 1) ? wh[k >> 1] >> 8 : wh[k >> 1];
                a0[k] = l & 0x000F000Fu; a2[k] = l & 0x00F000F0u;
                a1[k] = h & 0x000F000Fu; a3[k] = h & 0x00F000F0u;
              } else {
                a0[k] = wl[k] & 0x00FF00FFu; a2[k] = (wl[k] >> 8) & 0x00FF00FFu;
                a1[k] = wh[k] & 0x00FF00FFu; a3[k] = (wh[k] >> 8) & 0x00FF00FFu;
              }
            }
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
              const uint32_t bb[8] = {bf[nt][0].x, bf[nt][0].y, bf[nt][0].z, bf[nt][0].w, bf[nt][1].x, bf[nt][1].y, bf[nt][1].z, bf[nt][1].w};
              float (&y)[4] = acc[tp][nt];
              if constexpr (GS != 32) {
                float d[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int k = 0; k < 4; ++k) mma_f16_16816(d, a0[k], a1[k], a2[k], a3[k], bb[2 * k], bb[2 * k + 1]);
                y[0] = fmaf(s_lo[0], d[0], y[0]); y[1] = fmaf(s_lo[0], d[1], y[1]);
                y[2] = fmaf(s_hi[0], d[2], y[2]); y[3] = fmaf(s_hi[0], d[3], y[3]);
              } else {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                  float d[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                  for (int k = 2 * h; k < 2 * h + 2; ++k) mma_f16_16816(d, a0[k], a1[k], a2[k], a3[k], bb[2 * k], bb[2 * k + 1]);
                  if (h == 0 || k0 + (ch * kGC + wk) * 64 + 32 < p.K) {   // the last half group may not exist
                    y[0] = fmaf(s_lo[h], d[0], y[0]); y[1] = fmaf(s_lo[h], d[1], y[1]);
                    y[2] = fmaf(s_hi[h], d[2], y[2]); y[3] = fmaf(s_hi[h], d[3], y[3]);
                  }
                }
              }
            }
          }
        }
      }
      // bias term of this stage: a tile's is one warp's turn
#pragma unroll
      for (int tp = 0; tp < kTPW; ++tp) {
        if (((ch + tp * (kWK / kTPW)) % kWK) == wk && (tp * kWR + wr) * 16 < b.n) {
          const uint32_t ba = sa + kRB * kSBP + tp * (kWR * 16 * kSBP);
#pragma unroll
          for (int sub = 0; sub < SUBS; ++sub) {
            // biases of (scale) groups 8 sub + 2 t, + 1 of rows g and g + 8; groups behind K count as 0
            const int i0 = SUBS * 8 * ch + 8 * sub + 2 * t, lim = (klen + (GS == 32 ? 31 : 63)) / (GS == 32 ? 32 : 64);
            uint32_t r[2] = {0u, 0u};
            if (i0 < lim) {
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                const uint32_t q = ba + h * 8 * kSBP + (GS == 128 ? 2 * t : 2 * (8 * sub + 2 * t));
                const uint32_t lo = lds_u16(q), hi = GS == 128 ? lo : (i0 + 1 < lim ? lds_u16(q + 2) : 0u);
                r[h] = lo | (hi << 16);
              }
            }
#pragma unroll
            for (int nt = 0; nt < NT; ++nt)
#pragma unroll
              for (int k = 0; k < 3; ++k)
                mma_bf16_1688(acc[tp][nt], r[0], r[1], lds_u32(xb_s + (uint32_t)((((ch * SUBS + sub) * 3 + k) * NT + nt) * 128 + g * 16 + 4 * t)));
          }
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(empty + 8 * st);
      advance();
    }

    // ---- the block's sums: over the warps of a tile in shared memory, over the cluster through distributed shared memory ----
    mbar_wait(full + 8 * st, ph, polls, 4);
    if (pw[0] == 0) pw[1 + (rxn & 1)] = 1;                    // seen by all consumers behind the barrier that they meet at next
    unsigned char* red = smem + (size_t)st * GE::STAGE;       // [wk][tile][lane] float4, one token tile at a time
    const int oc = 512 / cs;                                  // outputs of a token tile that one CTA finishes
    if (cs > 1 && rxn == 0) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    float vout[NT];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      if (nt > 0) consumers_sync();
#pragma unroll
      for (int tp = 0; tp < kTPW; ++tp)
        *(float4*)(red + ((size_t)(wk * 4 + tp * kWR + wr) * 32 + lane) * 16) = make_float4(acc[tp][nt][0], acc[tp][nt][1], acc[tp][nt][2], acc[tp][nt][3]);
      consumers_sync();
      float s = 0.f;
#pragma unroll
      for (int k = 0; k < kWK; ++k) s += ((const float*)red)[k * 512 + tid];
      // thread = (tile, lane, component) of the accumulator layout
      const int col = nt * 8 + 2 * ((tid >> 2) & 3) + (tid & 1);
      vout[nt] = s * s_ts[col];
      if (cs > 1) {
        const uint32_t owner = (uint32_t)(tid / oc);
        float* slot = recv + ((size_t)((rxn & 1) * cs + crank) * NT + nt) * oc + tid % oc;
        st_cluster_f32(map_to_rank(smem_u32(slot), owner), vout[nt]);
      }
    }
    const int out = pw[1 + (rxn & 1)];                        // (the same for all: the next block writes the other word)
    __syncwarp();
    if (lane == 0) mbar_arrive(empty + 8 * st);
    advance();
    int o = tid;
    bool mine = true;
    if (cs > 1) {
      // every warp tells every CTA of the cluster that its part has been written
      if (lane < cs && !out) {                                // (no arrival: the peers' waits run out too)
        const uint32_t rb = map_to_rank(rx + 8 * (rxn & 1), (uint32_t)lane);
        asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(rb) : "memory");
      }
      if (!out) mbar_wait<true>(rx + 8 * (rxn & 1), (uint32_t)((rxn >> 1) & 1), polls, 5);
      mine = tid < oc;
      o = crank * oc + tid;
      if (mine) {
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
          float s = 0.f;
          for (int r = 0; r < cs; ++r) s += recv[((size_t)((rxn & 1) * cs + r) * NT + nt) * oc + tid];
          vout[nt] = s;
        }
      }
    }
    // oc is a multiple of 32 lanes and of a lane's 4 components: a warp stores or does not
    const bool good = !out && (cs == 1 || pw[0] != 0);
    if (mine) {
      const int row = (o >> 7) * 16 + ((o & 127) >> 4) + 8 * ((o >> 1) & 1);
      void* ym = QB_SEL4(p.y, b.mi);
      const int64_t ldy = QB_SEL4(p.ldy, b.mi);
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        const int col = nt * 8 + 2 * ((o >> 2) & 3) + (o & 1);
        if (p.x_f32) {
          const float s = vout[nt] + __shfl_xor_sync(0xffffffffu, vout[nt], 1);   // high and low part of one token
          if (!(o & 1) && (col >> 1) < p.M && row < b.n && good) ((float*)ym)[(int64_t)(col >> 1) * ldy + b.row + row] = s;
        } else if (col < p.M && row < b.n && good) {
          ((uint16_t*)ym)[(int64_t)col * ldy + b.row + row] = f32_to_bf16_bits(vout[nt]);
        }
      }
    }
    ++rxn;
    if (out) break;
  }
  if (cs > 1) {
    if (rxn == 0) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    cluster_sync_all();
  }
}

size_t smem_bytes(int stage, int ns, int gc, int nt, int ct, int cs, int gs) {
  return (size_t)ns * stage + (size_t)gc * 128 * nt * ct + (size_t)((gc + kGC - 1) / kGC) * (gs == 32 ? 2 : 1) * 3 * nt * 128 +
         (cs > 1 ? (size_t)nt * 4096 : 0) + 128 + 32 * nt + 16 * ns + 32;
}

// Cluster size, stages and shared memory of a launch with `cols` activation columns; false when the activations do not fit.
bool plan(F16K& p, int cols, int bits, int gs, int* nt_out, size_t* smem_out) {
  const int nt = cols <= 8 ? 1 : (cols <= 16 ? 2 : 4);
  int ct = 8;
  if (nt == 1) { ct = 1; while (ct < cols) ct *= 2; }
  const int stage = bits == 4 ? Geo<4>::STAGE : Geo<8>::STAGE;
  const size_t budget = (size_t)227 * 1024;
  const int groups = (p.K + 63) / 64;
  int cs = 1, ns = 0, gc = groups;
  for (; cs <= 8; cs *= 2) {
    gc = (groups + cs - 1) / cs;
    if (gs == 128) gc = (gc + 1) / 2 * 2;
    for (ns = 5; ns >= 2; --ns)
      if (smem_bytes(stage, ns, gc, nt, ct, cs, gs) <= budget) break;
    if (ns >= (bits == 4 ? 3 : 2)) break;
  }
  if (cs > 8) return false;
  p.cluster = cs; p.gc = gc; p.ct = ct; p.stages = ns;
  *nt_out = nt;
  *smem_out = smem_bytes(stage, ns, gc, nt, ct, cs, gs);
  return true;
}

template <int BITS, int NT, int GS>
cudaError_t launch_inst(const F16K& p, size_t smem, cudaStream_t st) {
  auto kern = qmv_f16_kernel<BITS, NT, GS>;
  static bool attr_done[64] = {};
  static int clusters_of[64][4] = {};   // co-resident clusters of 2, 4, 8 CTAs at the full footprint of the instantiation; -1: none
  int dev = 0;
  cudaGetDevice(&dev);
  const int di = (dev >= 0 && dev < 64) ? dev : 0;
  const int ci = p.cluster == 1 ? 0 : (p.cluster == 2 ? 1 : (p.cluster == 4 ? 2 : 3));
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(kThreads);
  {
    std::lock_guard<std::mutex> lk(setup_mutex());   // first use on a device, from any thread
    if (!attr_done[di] || di != dev) {
      const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
      if (e != cudaSuccess) return e;
      note_reader((const void*)kern);
      attr_done[di] = true;
    }
    if (p.cluster > 1 && (clusters_of[di][ci] == 0 || di != dev)) {
      const int n = sm_count() / p.cluster;
      cfg.gridDim = dim3(n * p.cluster);
      cfg.dynamicSmemBytes = (size_t)227 * 1024;
      attr[1].val.clusterDim.x = p.cluster;
      cfg.attrs = &attr[1];
      cfg.numAttrs = 1;
      int q = 0;
      if (cudaOccupancyMaxActiveClusters(&q, kern, &cfg) != cudaSuccess) { (void)cudaGetLastError(); q = 0; }
      clusters_of[di][ci] = q < 1 ? -1 : (q < n ? q : n);
    }
  }
  int ncl = p.cluster > 1 ? clusters_of[di][ci] : sm_count();
  if (ncl < 1) return cudaErrorInvalidConfiguration;
  const int most = (p.row0[p.nmat] + 7) / 8;           // a cluster has at least 8 rows
  ncl = ncl < most ? ncl : most;
  cfg.gridDim = dim3(ncl * p.cluster);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  attr[1].val.clusterDim.x = p.cluster;
  cfg.attrs = attr;
  cfg.numAttrs = p.cluster > 1 ? 2 : 1;
  return p.cluster > 1 ? launch_clusters(cfg, kern, p) : cudaLaunchKernelEx(&cfg, kern, p);
}
template <int BITS, int NT>
cudaError_t launch_gs(const F16K& p, int gs, size_t smem, cudaStream_t st) {
  if (gs == 32) return launch_inst<BITS, NT, 32>(p, smem, st);
  if (gs == 128) return launch_inst<BITS, NT, 128>(p, smem, st);
  return launch_inst<BITS, NT, 64>(p, smem, st);
}
template <int BITS>
cudaError_t launch_nt(const F16K& p, int nt, int gs, size_t smem, cudaStream_t st) {
  if (nt == 1) return launch_gs<BITS, 1>(p, gs, smem, st);
  if (nt == 2) return launch_gs<BITS, 2>(p, gs, smem, st);
  return launch_gs<BITS, 4>(p, gs, smem, st);
}

}  // namespace

int qmv_f16_error_code() {
  int v = 0;
  cudaMemcpyFromSymbol(&v, g_f16_error, sizeof(int));
  return v ? 200 + v : 0;
}
void qmv_f16_error_reset() {
  const int zero = 0;
  cudaMemcpyToSymbol(g_f16_error, &zero, sizeof(int));
}

bool qmv_f16_supported(const QmmArgs& a) {
  if (!a.transpose || a.nbatch != 1) return false;
  if (a.bits != 4 && a.bits != 8) return false;
  if (a.gs != 32 && a.gs != 64 && a.gs != 128) return false;
  if (a.x_dtype != QB200_BFLOAT16 && a.x_dtype != QB200_FLOAT32) return false;
  if (a.K % a.gs != 0 || a.K <= 0 || a.K > (1 << 20) || a.N <= 0 || a.N > (1 << 24) || a.M <= 0) return false;
  if ((((uintptr_t)a.w) & 15) != 0 || (a.ldw * 4) % 16 != 0 || (a.K * a.bits / 8) % 16 != 0) return false;
  if ((((uintptr_t)a.s) & 15) != 0 || (((uintptr_t)a.b) & 15) != 0) return false;
  if (a.ldw < 0 || a.lds < 0) return false;
  F16K p;
  p.K = (int)a.K;
  int nt;
  size_t smem;
  const int per = a.x_dtype == QB200_FLOAT32 ? 16 : 32;
  const int cols = (int)(a.M < per ? a.M : per) * (a.x_dtype == QB200_FLOAT32 ? 2 : 1);
  return plan(p, cols, a.bits, a.gs, &nt, &smem);
}

// `count` (<= 4) weight matrices applied to the same activations in one launch.  Every entry must have passed
// qmv_f16_supported and share x, M, K, dtype, bits and group size with the first.  More columns than a launch holds run in
// blocks that stream the weights again (out of L2 where they fit).
cudaError_t launch_qmv_f16_multi(const QmmArgs* a, int count, cudaStream_t st) {
  F16K p;
  p.nmat = count;
  int rows = 0;
  for (int i = 0; i < kMaxMat; ++i) {
    const QmmArgs& q = a[i < count ? i : 0];
    p.w[i] = q.w + q.wb.offset(0);
    p.s[i] = (const uint16_t*)q.s + q.sb.offset(0);
    p.b[i] = (const uint16_t*)q.b + q.sb.offset(0);
    p.N[i] = i < count ? (int)q.N : 0;
    p.ldw[i] = q.ldw; p.lds[i] = q.lds; p.ldy[i] = q.ldy;
    p.row0[i] = rows;
    rows += p.N[i];
  }
  p.row0[kMaxMat] = rows;
  p.K = (int)a[0].K;
  p.ldx = a[0].ldx;
  p.x_f32 = a[0].x_dtype == QB200_FLOAT32;
  p.polls = wait_polls() == 0 ? kPolls : (wait_polls() > 0 ? wait_polls() : 0);
  const int esz = p.x_f32 ? 4 : 2;
  const int64_t per = p.x_f32 ? 16 : 32;
  for (int64_t m0 = 0; m0 < a[0].M; m0 += per) {
    p.x = (const char*)a[0].x + (a[0].xb.offset(0) + m0 * a[0].ldx) * esz;
    for (int i = 0; i < kMaxMat; ++i) {
      const QmmArgs& q = a[i < count ? i : 0];
      p.y[i] = (char*)q.y + (q.yb.offset(0) + m0 * q.ldy) * esz;
    }
    p.M = (int)((a[0].M - m0) < per ? (a[0].M - m0) : per);
    p.early = m0 > 0 || weights_settled(st);   // (behind the first block: that block's launch is what comes before)
    int nt;
    size_t smem;
    if (!plan(p, p.M * (p.x_f32 ? 2 : 1), a[0].bits, a[0].gs, &nt, &smem)) return cudaErrorInvalidConfiguration;
    const cudaError_t e = a[0].bits == 4 ? launch_nt<4>(p, nt, a[0].gs, smem, st) : launch_nt<8>(p, nt, a[0].gs, smem, st);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}
cudaError_t launch_qmv_f16(const QmmArgs& a, cudaStream_t st) { return launch_qmv_f16_multi(&a, 1, st); }

}  // namespace qb
