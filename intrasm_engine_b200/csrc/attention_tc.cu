// The SDDMM -> SpMM chain of masked attention in one launch over all heads, fp32 in and out:
//   out[h, i, :] = sum over the mask's positions (i, j) of dot(q[h, i], k[h, j]) * v[h, j, :]
//
// Called operator by operator the chain takes a tensor-core SDDMM and a CUDA-core SpMM per head (18 + 22 us
// at 4096 x 4096, 5 %, d = 64; 30 us a head over two streams) plus a few launches' host time per head: the
// SpMM is bound by gathering a row of v per position through L2.  Here both products are dense tiles on
// the tensor cores and the mask is applied in between, in tensor memory, flash-attention style: scores
// never leave the SM and v is read once per 128 rows.
//
// fp32 accuracy: operands are split into TF32 head and tail (x = hi + lo) and three of the four products
// are kept, as in sddmm_tc.cu.  The tensor core truncates when it adds to an accumulator, which would bias
// a sum over thousands of positions (2e-6 of the result, measured); a tile's 64 keys are therefore added to
// fp32 registers with ordinary rounding before the next tile: as accurate as the CUDA-core sum (2.6e-7).
//
//   prepare kernel   k and v (transposed) as hi / lo planes that TMA can load; looks for values of v that are not
//                    finite and clears the counters of the bands' pieces
//   main kernel      one persistent CTA per SM over a contiguous run of (head, 128-row band, key tile)
//     warp 0         TMA producer: k planes and v planes of a key tile in two rings (k is free again after S, a
//                    tile earlier than v: one ring for both left loads too little time, 2600 cycles a tile)
//     warp 1         issues S(t) = Q K(t)^T, warp 2 O(t) = P(t) V(t); A operands (Q, P) in tensor memory.  Two
//                    warps because a thread that issues for a busy tensor pipe pays 200-300 cycles for every
//                    barrier it waits on, completed or not, and 100 for a commit: one for both products took
//                    2740 cycles a tile, of which the pipe needs 1540
//     warps 4-11     read S, keep the mask's positions, write P hi / lo over it; add the O of the tile before to
//                    registers.  Two warps per tensor-memory quarter share a tile's columns: the tensor pipe
//                    only has S(t + 1) to do until P(t) is there, so the time from S to P is what counts
//                    (one warp per quarter and tile, taking turns: 2900 cycles a tile)
// The runs are equal shares of all tiles; with fewer bands than SMs, every band is cut into the same number of equal pieces
// instead (cta_count).  The pieces of a band meet in a workspace and are added in order by whichever comes last.
//
// 24 heads x 4096 x 4096 at 5 %, d 64: 499 us in the first tenth of a second (1965 MHz), 547 to 565 us sustained (1430 to 1470
// MHz, at the power limit); head by head over two streams 723 us.  6 heads x 1003 x 1003 at 10 %, d 80: 30.7 us against 147.
// Which masks are faster one way or the other: iex_attention_f32_prefers below.
//
// Values of v at masked-out positions must not count even if they are not finite.  Zero times such a value is
// not zero, so the prepare kernel looks for them and the (rare) heads that have some are summed position
// by position.
//
// Every mbarrier wait is bounded, as in tc_fused.cu.
#include <cuda.h>

#include <algorithm>
#include <cmath>
#include <mutex>

#include "common.cuh"
#include "tc_ptx.cuh"

namespace iex {
namespace tc {

int make_map_f32(CUtensorMap* map, const void* base, long long rows, long long cols, int box_rows);  // tc_fused.cu

namespace {

constexpr int kThreads = 384;
constexpr int kMaxStages = 6;      // of either ring
constexpr int kBars = 4 * kMaxStages + 8;
constexpr int kBarBytes = 8 * kBars + 16;
constexpr int kBudget = (227 * 1024 - 1024 - kBarBytes) & ~1023;

struct AttnParams {
  int heads, m, n, d, dv;
  int parts, dvt;                // a head's columns of v in parts of DVP (wide heads: two), dvt = parts * DVP
  int bands, tiles, mp;          // 128-row bands, key tiles per band, rows of the mask words
  int np;                        // row length of the transposed v planes
  int total;                     // heads * parts * bands * tiles
  int k_stages, v_stages;
  const uint32_t* bits;          // [key words][mp]
  const float* q;
  const float* k;
  const float* v;
  float* out;
  const int* row_offsets;
  const int* cols;
  float4* partials;              // [2 * CTAs][dvp / 4][128]: sums of a CTA's first and last band where they are cut
  int* counters;                 // [bands of all heads and parts][8]: pieces of a band that are there, per warp
  const int* flags;              // [heads][flag_blocks]: values of v that are not finite
  int flag_blocks;
  int* status;
};

__device__ __forceinline__ int range_begin(int c, int total, int ctas) {
  return static_cast<int>(static_cast<long long>(c) * total / ctas);
}

// The CTA whose range holds tile t.
__device__ __forceinline__ int cta_of(int t, int total, int ctas) {
  return static_cast<int>(((t + 1ll) * ctas - 1) / total);
}

// TF32 head of x, rounded half away from zero, by integer arithmetic on the sign-magnitude bits.
__device__ __forceinline__ uint32_t tf32_head(uint32_t x) { return (x + 0x1000u) & 0xffffe000u; }

__device__ __forceinline__ void umma_tf32_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc,
                                             uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem_d),
      "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
      "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// Rows [row0, row0 + 32) of one head, position by position (a warp; see the note on values that are not finite).
__device__ __noinline__ void rows_by_position(const AttnParams& p, int head, int row0, int lane) {
  const float* q = p.q + static_cast<size_t>(head) * p.m * p.d;
  const float* k = p.k + static_cast<size_t>(head) * p.n * p.d;
  const float* v = p.v + static_cast<size_t>(head) * p.n * p.dv;
  for (int r = row0; r < row0 + 32 && r < p.m; ++r) {
    float acc[4] = {0.f, 0.f, 0.f, 0.f};  // dv <= 128
    for (int e = p.row_offsets[r]; e < p.row_offsets[r + 1]; ++e) {
      const int j = p.cols[e];
      float s = 0.f;
      for (int c = lane; c < p.d; c += 32) s = fmaf(q[static_cast<size_t>(r) * p.d + c], k[static_cast<size_t>(j) * p.d + c], s);
      for (int x = 16; x >= 1; x >>= 1) s += __shfl_xor_sync(0xffffffffu, s, x);
      for (int i = 0; i < 4; ++i)
        if (lane + 32 * i < p.dv) acc[i] = fmaf(s, v[static_cast<size_t>(j) * p.dv + lane + 32 * i], acc[i]);
    }
    for (int i = 0; i < 4; ++i)
      if (lane + 32 * i < p.dv) p.out[(static_cast<size_t>(head) * p.m + r) * p.dv + lane + 32 * i] = acc[i];
  }
}

// kDA: 32-float atoms of d (rounded up); KT: keys per tile; kOut: 16-float pieces of dv (rounded up)
template <int kDA, int KT, int kOut>
__global__ void __launch_bounds__(kThreads, 1)
attention_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v, const AttnParams p) {
  constexpr int DP = kDA * 32, DVP = kOut * 16;
  constexpr uint32_t kQHi = 0, kQLo = DP, kS = 2 * DP, kO = 2 * DP + 4 * KT;
  static_assert(2 * DP + 4 * KT + 2 * DVP <= 512, "tensor memory");
  constexpr uint32_t kKPlane = KT * DP * 4, kVPlane = KT * DVP * 4;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* base_ptr = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t bar = base + kBudget;
  auto k_full = [&](int s) { return bar + 8u * s; };
  auto k_empty = [&](int s) { return bar + 8u * (kMaxStages + s); };
  auto v_full = [&](int s) { return bar + 8u * (2 * kMaxStages + s); };
  auto v_empty = [&](int s) { return bar + 8u * (3 * kMaxStages + s); };
  const uint32_t v_base = base + p.k_stages * 2u * kKPlane;
  constexpr uint32_t kB0 = 32u * kMaxStages;
  auto s_full = [&](int b) { return bar + kB0 + 8u * b; };
  auto p_full = [&](int b) { return bar + kB0 + 16u + 8u * b; };
  auto pv_done = [&](int b) { return bar + kB0 + 32u + 8u * b; };
  const uint32_t q_full = bar + kB0 + 48u, seg_done = bar + kB0 + 56u;
  volatile uint32_t* tmem_ptr = reinterpret_cast<volatile uint32_t*>(base_ptr + kBudget + 8 * kBars);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_ptr + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < 4 * kMaxStages; ++s) mbar_init(bar + 8u * s, 1);
    for (int b = 0; b < 2; ++b) {
      mbar_init(s_full(b), 1);
      mbar_init(p_full(b), 8);
      mbar_init(pv_done(b), 1);
    }
    mbar_init(q_full, 8);
    mbar_init(seg_done, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(bar + 8u * kBars), "r"(512u)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem = *tmem_ptr;
  grid_dependency_wait();
  grid_launch_dependents();

  const int r0 = range_begin(blockIdx.x, p.total, gridDim.x), r1 = range_begin(blockIdx.x + 1, p.total, gridDim.x);

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (elect_one()) {
      asm volatile("prefetch.tensormap [%0];" ::"l"(&map_k) : "memory");
      asm volatile("prefetch.tensormap [%0];" ::"l"(&map_v) : "memory");
      int sk = 0, sv = 0;
      uint32_t phk = 0, phv = 0;
      for (int r = r0; r < r1; ++r) {
        const int item = r / p.tiles, t = r - item * p.tiles, unit = item / p.bands, head = unit / p.parts;
        if (!mbar_wait(k_empty(sk), phk ^ 1u, abort_flag, p.status, 32)) break;
        mbar_arrive_expect_tx(k_full(sk), 2 * kKPlane);
#pragma unroll
        for (int pl = 0; pl < 2; ++pl)
#pragma unroll
          for (int a = 0; a < kDA; ++a)
            tma_load_2d(base + (2 * sk + pl) * kKPlane + a * (KT * 128), &map_k, k_full(sk), a * 32,
                        (pl * p.heads + head) * p.n + t * KT);
        if (!mbar_wait(v_empty(sv), phv ^ 1u, abort_flag, p.status, 32)) break;
        mbar_arrive_expect_tx(v_full(sv), 2 * kVPlane);
#pragma unroll
        for (int pl = 0; pl < 2; ++pl)
#pragma unroll
          for (int a = 0; a < KT / 32; ++a)
            tma_load_2d(v_base + (2 * sv + pl) * kVPlane + a * (DVP * 128), &map_v, v_full(sv), t * KT + a * 32,
                        pl * p.heads * p.dvt + unit * DVP);
        if (++sk == p.k_stages) { sk = 0; phk ^= 1u; }
        if (++sv == p.v_stages) { sv = 0; phv ^= 1u; }
      }
      if (*abort_flag)
        for (uint32_t i = 0; i < 2048u; ++i) __nanosleep(100);
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------------------ S = Q K^T
    if (elect_one()) {
      constexpr uint32_t idesc = (1u << 4) | (2u << 7) | (2u << 10) | (static_cast<uint32_t>(KT >> 3) << 17) | (8u << 24);
      int st = 0;
      uint32_t ph = 0, seg = 0;
      bool ok = true;
      for (int r = r0; r < r1 && ok; ++seg) {
        const int seg_end = min(r1, (r / p.tiles + 1) * p.tiles);
        if (!mbar_wait(q_full, seg & 1u, abort_flag, p.status, 20)) break;
        for (; r < seg_end; ++r) {
          const int g = r - r0, b = g & 1;
          if (!mbar_wait(k_full(st), ph, abort_flag, p.status, 20) ||
              !mbar_wait(pv_done(b), ((g >> 1) & 1u) ^ 1u, abort_flag, p.status, 20)) { ok = false; break; }
          tcgen05_fence_after();
          const uint32_t k_hi = base + 2 * st * kKPlane, d = tmem + kS + b * 2 * KT;
          // small terms first: lo * hi', hi * lo', then hi * hi'
#pragma unroll
          for (int pr = 0; pr < 3; ++pr)
#pragma unroll
            for (int a = 0; a < kDA; ++a) {
              const uint64_t bd = smem_desc(k_hi + (pr == 1 ? kKPlane : 0u) + a * (KT * 128), 16, 1024);
#pragma unroll
              for (int ks = 0; ks < 4; ++ks)
                umma_tf32_ts(d, tmem + (pr == 0 ? kQLo : kQHi) + a * 32 + ks * 8, desc_advance(bd, ks * 32), idesc,
                             (pr | a | ks) != 0 ? 1u : 0u);
            }
          umma_commit(s_full(b));
          umma_commit(k_empty(st));
          if (++st == p.k_stages) { st = 0; ph ^= 1u; }
        }
      }
    }
    __syncwarp();
  } else if (warp == 2) {
    // ------------------------------------------------------------------ O = P V
    if (elect_one()) {
      constexpr uint32_t idesc = (1u << 4) | (2u << 7) | (2u << 10) | (static_cast<uint32_t>(DVP >> 3) << 17) | (8u << 24);
      int st = 0;
      uint32_t ph = 0;
      for (int r = r0; r < r1; ++r) {
        const int g = r - r0, b = g & 1;
        // P(g) also says that O(g - 2) has been read: every warp adds it before it writes P(g)
        if (!mbar_wait(v_full(st), ph, abort_flag, p.status, 20) ||
            !mbar_wait(p_full(b), (g >> 1) & 1u, abort_flag, p.status, 20)) break;
        tcgen05_fence_after();
        const uint32_t v_hi = v_base + 2 * st * kVPlane, d = tmem + kO + b * DVP, pp = tmem + kS + b * 2 * KT;
#pragma unroll
        for (int pr = 0; pr < 3; ++pr)
#pragma unroll
          for (int a = 0; a < KT / 32; ++a) {
            const uint64_t bd = smem_desc(v_hi + (pr == 1 ? kVPlane : 0u) + a * (DVP * 128), 16, 1024);
#pragma unroll
            for (int ks = 0; ks < 4; ++ks)
              umma_tf32_ts(d, pp + (pr == 0 ? KT : 0) + a * 32 + ks * 8, desc_advance(bd, ks * 32), idesc,
                           (pr | a | ks) != 0 ? 1u : 0u);
          }
        umma_commit(pv_done(b));
        umma_commit(v_empty(st));
        if (r + 1 == r1 || (r + 1) % p.tiles == 0) umma_commit(seg_done);  // a band's last tile
        if (++st == p.v_stages) { st = 0; ph ^= 1u; }
      }
    }
    __syncwarp();
  } else if (warp >= 4) {
    // ------------------------------------------------------------------ mask and sums
    const int wg = warp >= 8 ? 1 : 0, q4 = warp & 3;
    const uint32_t lanes = tmem + (static_cast<uint32_t>(q4 * 32) << 16);
    const int row_local = q4 * 32 + lane;
    bool ok = true;
    uint32_t seg = 0;
    for (int r = r0; r < r1 && ok; ++seg) {
      const int item = r / p.tiles, unit = item / p.bands, band = item - unit * p.bands;
      const int head = unit / p.parts, col0 = (unit - head * p.parts) * DVP;
      const int t_begin = r - item * p.tiles;
      const int seg_end = min(r1, (item + 1) * p.tiles);
      const int row = band * 128 + row_local;
      {  // this warp group's half of the band's q columns into tensor memory
        constexpr int kHalf = DP / 2;
        const float* src = p.q + (static_cast<size_t>(head) * p.m + row) * p.d + wg * kHalf;
        uint32_t x[kHalf];
#pragma unroll
        for (int j = 0; j < kHalf / 4; ++j) {
          float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
          if (row < p.m && wg * kHalf + 4 * j < p.d) f = __ldg(reinterpret_cast<const float4*>(src) + j);
          x[4 * j] = __float_as_uint(f.x);
          x[4 * j + 1] = __float_as_uint(f.y);
          x[4 * j + 2] = __float_as_uint(f.z);
          x[4 * j + 3] = __float_as_uint(f.w);
        }
        // the tensor core is done with the previous band (all its tiles, both groups')
        if (seg > 0 && !mbar_wait(seg_done, (seg - 1u) & 1u, abort_flag, p.status, 32)) { ok = false; break; }
        __syncwarp();
        tcgen05_fence_after();
#pragma unroll
        for (int h = 0; h < kHalf / 16; ++h) {
          uint32_t hi[16], lo[16];
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            hi[j] = tf32_head(x[16 * h + j]);
            lo[j] = __float_as_uint(__uint_as_float(x[16 * h + j]) - __uint_as_float(hi[j]));
          }
          tmem_st16(lanes + kQHi + wg * kHalf + h * 16, hi);
          tmem_st16(lanes + kQLo + wg * kHalf + h * 16, lo);
        }
        tmem_wait_st();
        tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(q_full);
      }
      // this warp group's half of a tile's keys and of the output columns
      constexpr int kKeys = KT / 2, kCols = DVP / 2;
      float acc[kCols];
#pragma unroll
      for (int j = 0; j < kCols; ++j) acc[j] = 0.f;
      auto add_tile = [&](int g) -> bool {  // O of tile g
        const int b = g & 1;
        if (!mbar_wait(pv_done(b), (g >> 1) & 1u, abort_flag, p.status, 20)) return false;
        __syncwarp();
        tcgen05_fence_after();
        uint32_t o[kCols];
#pragma unroll
        for (int h = 0; h < kCols / 16; ++h) tmem_ld16(lanes + kO + b * DVP + wg * kCols + h * 16, &o[16 * h]);
        tmem_wait_ld();
#pragma unroll
        for (int j = 0; j < kCols; ++j) acc[j] += __uint_as_float(o[j]);
        tcgen05_fence_before();
        return true;
      };
      const int tiles_here = seg_end - r, g0 = r - r0;
      // the row's mask bits of this half of a tile: a word, or half of one
      const uint32_t* bits = p.bits + static_cast<size_t>(t_begin) * (KT / 32) * p.mp + (KT == 64 ? wg * p.mp : 0) + band * 128 + row_local;
      auto mask_of = [&](int t) -> uint32_t {
        const uint32_t w = t < tiles_here ? __ldg(bits + static_cast<size_t>(t) * (KT / 32) * p.mp) : 0u;
        return KT == 64 ? w : w >> (wg * 16);
      };
      uint32_t w = mask_of(0);
      for (int t = 0; t < tiles_here; ++t) {
        const int g = g0 + t, b = g & 1;
        const uint32_t next = mask_of(t + 1);
        if (!mbar_wait(s_full(b), (g >> 1) & 1u, abort_flag, p.status, 20)) { ok = false; break; }
        __syncwarp();
        tcgen05_fence_after();
        const uint32_t s_addr = lanes + kS + b * 2 * KT + wg * kKeys;
        uint32_t x[kKeys];
#pragma unroll
        for (int h = 0; h < kKeys / 16; ++h) tmem_ld16(s_addr + h * 16, &x[16 * h]);
        tmem_wait_ld();
#pragma unroll
        for (int h = 0; h < kKeys / 16; ++h) {
          uint32_t hi[16], lo[16];
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const uint32_t v = (w & (1u << (16 * h + j))) ? x[16 * h + j] : 0u;
            hi[j] = tf32_head(v);
            lo[j] = __float_as_uint(__uint_as_float(v) - __uint_as_float(hi[j]));
          }
          tmem_st16(s_addr + h * 16, hi);
          tmem_st16(s_addr + KT + h * 16, lo);
        }
        tmem_wait_st();
        tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(p_full(b));
        if (t > 0 && !add_tile(g - 1)) { ok = false; break; }
        w = next;
      }
      if (!ok || !add_tile(g0 + tiles_here - 1)) { ok = false; break; }
      bool finite = true;
      for (int i = lane; i < p.flag_blocks; i += 32) finite = finite && __ldg(p.flags + head * p.flag_blocks + i) == 0;
      finite = __all_sync(0xffffffffu, finite);
      bool write = finite;
      if (finite && tiles_here != p.tiles) {
        // A band cut between CTAs: this piece goes to the workspace, and the warp that finds all the others there adds them
        // up in the order of the keys.
        constexpr int kQuads = kCols / 4;
        const int first_tile = item * p.tiles;
        const int first = cta_of(first_tile, p.total, gridDim.x), last = cta_of(first_tile + p.tiles - 1, p.total, gridDim.x);
        const size_t mine = static_cast<size_t>(wg) * kQuads * 128 + row_local;
        float4* to = p.partials + (2 * blockIdx.x + (r == r0 ? 0 : 1)) * static_cast<size_t>(DVP / 4 * 128) + mine;
#pragma unroll
        for (int j = 0; j < kQuads; ++j)
          __stcg(to + j * 128, make_float4(acc[4 * j], acc[4 * j + 1], acc[4 * j + 2], acc[4 * j + 3]));
        __threadfence();
        __syncwarp();
        int there = 0;
        if (lane == 0) there = atomicAdd(p.counters + item * 8 + wg * 4 + q4, 1);
        write = __shfl_sync(0xffffffffu, there, 0) == last - first;
        if (write) {
          __threadfence();
#pragma unroll
          for (int j = 0; j < kCols; ++j) acc[j] = 0.f;
          for (int c = first; c <= last; ++c) {
            const int slot = 2 * c + (range_begin(c, p.total, gridDim.x) < first_tile ? 1 : 0);
            const float4* from = p.partials + slot * static_cast<size_t>(DVP / 4 * 128) + mine;
            float4 x[kQuads];
#pragma unroll
            for (int j = 0; j < kQuads; ++j) x[j] = __ldcg(from + j * 128);
#pragma unroll
            for (int j = 0; j < kQuads; ++j) {
              acc[4 * j] += x[j].x;
              acc[4 * j + 1] += x[j].y;
              acc[4 * j + 2] += x[j].z;
              acc[4 * j + 3] += x[j].w;
            }
          }
        }
      }
      if (write && row < p.m) {
        float* dst = p.out + (static_cast<size_t>(head) * p.m + row) * p.dv + col0 + wg * kCols;
#pragma unroll
        for (int j = 0; j < kCols / 4; ++j)
          if (col0 + wg * kCols + 4 * j < p.dv)
            reinterpret_cast<float4*>(dst)[j] = make_float4(acc[4 * j], acc[4 * j + 1], acc[4 * j + 2], acc[4 * j + 3]);
      }
      if (!finite && t_begin == 0 && wg == 0 && col0 == 0) rows_by_position(p, head, band * 128 + q4 * 32, lane);
      r = seg_end;
    }
  }
  tcgen05_fence_before();
  __syncthreads();
  if (warp == 1) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
}

constexpr int kPrepKeys = 64;

// Block (x, h): keys [64 x, +64) of head h as hi / lo planes.  k planes [2][heads * n][dp], v planes transposed,
// [2][heads * dvt][np].  The blocks of the last y zero the main kernel's counters.
__global__ void __launch_bounds__(256)
attention_prepare_kernel(const AttnParams p, int dp, float* __restrict__ k_planes, float* __restrict__ v_planes,
                         int* __restrict__ flags) {
  extern __shared__ float v_tile[];  // [64][dv + 1]
  grid_dependency_wait();
  grid_launch_dependents();
  if (static_cast<int>(blockIdx.y) == p.heads) {
    const int counters = p.heads * p.parts * p.bands * 8;
    for (int i = blockIdx.x * 256 + threadIdx.x; i < counters; i += gridDim.x * 256) p.counters[i] = 0;
    return;
  }
  const int head = blockIdx.y, key0 = blockIdx.x * kPrepKeys;
  const int keys = min(kPrepKeys, p.n - key0);  // may be <= 0 in the padding of the v planes
  const float* k = p.k + (static_cast<size_t>(head) * p.n + key0) * p.d;
  const float* v = p.v + (static_cast<size_t>(head) * p.n + key0) * p.dv;
  const size_t k_plane = static_cast<size_t>(p.heads) * p.n * dp;
  float* kd = k_planes + (static_cast<size_t>(head) * p.n + key0) * dp;
  const int d4 = dp / 4;
  for (int i = threadIdx.x; i < keys * d4; i += 256) {
    const int r = i / d4, c = (i - r * d4) * 4;
    float4 x = make_float4(0.f, 0.f, 0.f, 0.f), lo;
    if (c < p.d) x = __ldg(reinterpret_cast<const float4*>(k + static_cast<size_t>(r) * p.d + c));
    float4 hi = make_float4(__uint_as_float(tf32_head(__float_as_uint(x.x))), __uint_as_float(tf32_head(__float_as_uint(x.y))),
                            __uint_as_float(tf32_head(__float_as_uint(x.z))), __uint_as_float(tf32_head(__float_as_uint(x.w))));
    lo = make_float4(x.x - hi.x, x.y - hi.y, x.z - hi.z, x.w - hi.w);
    reinterpret_cast<float4*>(kd)[i] = hi;
    reinterpret_cast<float4*>(kd + k_plane)[i] = lo;
  }
  bool odd = false;  // a value whose head or product is not finite
  const int pitch = p.dv + 1;
  for (int i = threadIdx.x; i < keys * p.dv; i += 256) {
    const float x = __ldg(v + i);
    odd = odd || !(fabsf(x) < 1.7e38f);
    const int r = i / p.dv;
    v_tile[r * pitch + (i - r * p.dv)] = x;
  }
  const int any = __syncthreads_or(odd ? 1 : 0);
  if (threadIdx.x == 0) flags[head * gridDim.x + blockIdx.x] = any;
  const size_t v_plane = static_cast<size_t>(p.heads) * p.dvt * p.np;
  const int width = min(kPrepKeys, p.np - key0);
  for (int i = threadIdx.x; i < p.dvt * kPrepKeys; i += 256) {
    const int c = i / kPrepKeys, key = i % kPrepKeys;
    if (key >= width) continue;
    const float x = key < keys && c < p.dv ? v_tile[key * pitch + c] : 0.f;
    const float hi = __uint_as_float(tf32_head(__float_as_uint(x)));
    float* dst = v_planes + (static_cast<size_t>(head) * p.dvt + c) * p.np + key0 + key;
    dst[0] = hi;
    dst[v_plane] = x - hi;
  }
}

// bits[column / 32][row]; a position stored twice (a sum in the operators' terms) sets *repeated.
__global__ void __launch_bounds__(256)
attention_bits_kernel(int m, int mp, const int* __restrict__ row_offsets, const int* __restrict__ cols,
                      uint32_t* __restrict__ bits, uint32_t* __restrict__ repeated) {
  const int lane = threadIdx.x & 31;
  for (int r = blockIdx.x * 8 + (threadIdx.x >> 5); r < m; r += gridDim.x * 8)
    for (int e = __ldg(row_offsets + r) + lane; e < __ldg(row_offsets + r + 1); e += 32) {
      const int c = __ldg(cols + e);
      const uint32_t bit = 1u << (c & 31);
      if (atomicOr(bits + static_cast<size_t>(c >> 5) * mp + r, bit) & bit) *repeated = 1u;
    }
}

struct Shape {
  int da, kt, dp, dvp, parts, dvt, np, mp;
};

// Tensor memory holds q's planes (2 dp columns), two score tiles with their tails (4 kt) and two output
// tiles (2 dvp).
bool attention_shape(int heads, int m, int n, int d, int dv, Shape* s) {
  if (heads < 1 || m < 1 || n < 1 || d < 4 || dv < 4 || d % 4 != 0 || dv % 4 != 0 || d > 128 || dv > 128) return false;
  s->da = (d + 31) / 32;
  s->dvp = dv <= 32 ? 32 : dv <= 64 ? 64 : 96;
  s->parts = 1;
  if (s->da == 4 || dv > 96) {  // wide heads: v in parts of 64 columns, scores formed for each
    s->dvp = dv <= 32 ? 32 : 64;
    s->parts = (dv + s->dvp - 1) / s->dvp;
  }
  if (s->dvp == 96 && s->da < 3) s->da = 3;
  s->kt = s->da <= 2 ? 64 : 32;
  s->dp = s->da * 32;
  s->dvt = s->parts * s->dvp;
  s->np = (n + 31) / 32 * 32;
  s->mp = (m + 127) / 128 * 128;
  const long long tiles = static_cast<long long>(heads) * s->parts * ((m + 127) / 128) * ((n + s->kt - 1) / s->kt);
  return tiles < (1ll << 30) && 2ll * heads * n < (1ll << 30) && 2ll * heads * s->dvt < (1ll << 30) && heads <= 65000;
}

// One CTA per SM with an equal share of the tiles; with fewer bands than SMs, as many equal pieces of every band as
// fit on the chip, for a CTA that works on two bands pays for a second start (5 us), and no more than this
// root, since whoever comes last adds the pieces up alone.
int cta_count(int items, int tiles, int sms) {
  const int pieces = std::max(1, static_cast<int>(std::sqrt(1.5 * tiles)));
  return items >= sms ? sms : items * std::min(pieces, sms / items);
}

// Times in microseconds, fitted on B200 to 578 measurements: 1 to 32 heads, 256 to 16384 rows and keys, 32 to 128 columns,
// masks of 0.05 to 23 % stored positions, scattered or in a band.
//
// This kernel multiplies every tile, empty or not: m * n counts, not the positions.
double one_launch_us(int heads, int m, int n, const Shape& s, int sms) {
  const int bands = (m + 127) / 128, tiles = (n + s.kt - 1) / s.kt, items = heads * s.parts * bands;
  const int ctas = cta_count(items, tiles, sms);
  const double tile = (0.40 + 0.0032 * (s.da * s.kt + s.kt * s.dvp / 32)) * (s.kt == 32 ? 1.12 : 1.0);
  const double planes = static_cast<double>(heads) * n * (s.dp + s.dvt) * 12 / 6e6;
  return 13.0 + planes + (static_cast<long long>(items) * tiles + ctas - 1) / ctas * tile;
}

// SDDMM and SpMM head by head over two streams (pytorch/attention.py): 20 us of host time a head for the two launches, or
// what their gathers take, which follows the positions (a row of q.k and of v for each), and the dense tiles of the SDDMM
// where that is the tensor-core one.
double head_by_head_us(int heads, int m, int n, int d, int dv, int nnz) {
  auto row = [](int cols) { return cols <= 32 ? 32 : cols <= 64 ? 64 : 128; };
  double head = (0.6e-5 + 0.235e-6 * (row(d) + row(dv))) * nnz;
  if (iex_sddmm_f32_prefers_tc(m, d, n, nnz, 1)) head += 0.4e-6 * m * n;
  return std::max(28.0 + 19.5 * heads, 10.0 + heads * head);
}

size_t round256(size_t v) { return (v + 255) & ~static_cast<size_t>(255); }
int flag_blocks_of(int np) { return (np + kPrepKeys - 1) / kPrepKeys; }

template <int kDA, int KT, int kOut>
int launch_attention(const CUtensorMap& mk, const CUtensorMap& mv, AttnParams p, int ctas, cudaStream_t s) {
  constexpr int k_bytes = 2 * KT * kDA * 32 * 4, v_bytes = 2 * KT * kOut * 16 * 4;
  static_assert(2 * (k_bytes + v_bytes) <= kBudget, "two stages of each");
  p.k_stages = p.v_stages = 2;
  for (int left = kBudget - 2 * (k_bytes + v_bytes);;) {  // k first: it is asked for earlier
    if (p.k_stages <= p.v_stages && p.k_stages < kMaxStages && left >= k_bytes) { ++p.k_stages; left -= k_bytes; }
    else if (p.v_stages < kMaxStages && left >= v_bytes) { ++p.v_stages; left -= v_bytes; }
    else break;
  }
  auto kern = attention_kernel<kDA, KT, kOut>;
  static std::mutex mutex;
  static bool configured[64] = {};
  {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) dev = -1;
    std::lock_guard<std::mutex> lock(mutex);
    if (dev < 0 || dev >= 64 || !configured[dev]) {
      const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
      if (e != cudaSuccess) return static_cast<int>(e);
      if (dev >= 0 && dev < 64) configured[dev] = true;
    }
  }
  return launch_overlapped(kern, dim3(ctas), dim3(kThreads), static_cast<size_t>(227 * 1024), s, mk, mv, p);
}

}  // namespace
}  // namespace tc
}  // namespace iex

using namespace iex;
using namespace iex::tc;

extern "C" int iex_attention_f32_supported(int heads, int m, int n, int d, int dv) {
  Shape s;
  return attention_shape(heads, m, n, d, dv, &s) ? 1 : 0;
}

// One launch unless the operators are estimated a sixth shorter.  Where the line lies, measured (us, one launch / head by
// head): 4096 x 4096, 12 heads, d 80: 367 / 257 at 1 %, 367 / 307 at 2 %, 371 / 712 at 5 %; d 64: 211 / 265 from 0.05 to 2 %
// (the launches), 211 / 375 at 5 %; d 128: 741 / 256 at 1 %, 755 / 755 at 5 %, 761 / 1554 at 10 %.  16384 x 16384 with a band
// of 256, 8 heads, d 64: 2260 / 1425; with one of 1024: 2236 / 5026.  Of the 578 measurements the choice is the slower one by
// more than 10 % in three (14 % at most).
extern "C" int iex_attention_f32_prefers(int heads, int m, int n, int d, int dv, int nnz) {
  Shape s;
  if (!attention_shape(heads, m, n, d, dv, &s)) return 0;
  return one_launch_us(heads, m, n, s, std::min(sm_count(), kNumSMs)) <= 1.2 * head_by_head_us(heads, m, n, d, dv, nnz);
}

// Plan: one word (nonzero if a position is stored twice), then, 256 bytes on, the mask's bits.
extern "C" size_t iex_attention_plan_bytes(int m, int n) {
  if (m <= 0 || n <= 0) return 256;
  return 256 + static_cast<size_t>((n + 63) / 64 * 2) * ((m + 127) / 128 * 128) * 4;
}

extern "C" int iex_attention_plan_build(int m, int n, const int32_t* row_offsets, const int32_t* column_indices, void* plan,
                                        size_t bytes, void* stream) {
  if (m < 0 || n < 0 || !plan || !row_offsets || (reinterpret_cast<uintptr_t>(plan) & 255u)) return IEX_ERR_BAD_ARG;
  if (bytes < iex_attention_plan_bytes(m, n)) return IEX_ERR_TOO_LARGE;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const cudaError_t e = cudaMemsetAsync(plan, 0, iex_attention_plan_bytes(m, n), s);
  if (e != cudaSuccess) return static_cast<int>(e);
  if (m == 0 || n == 0) return IEX_OK;
  attention_bits_kernel<<<(m + 7) / 8 < 8 * kNumSMs ? (m + 7) / 8 : 8 * kNumSMs, 256, 0, s>>>(
      m, (m + 127) / 128 * 128, row_offsets, column_indices, static_cast<uint32_t*>(plan) + 64, static_cast<uint32_t*>(plan));
  return launch_status();
}

extern "C" size_t iex_attention_workspace_bytes(int heads, int m, int n, int d, int dv) {
  Shape s;
  if (!attention_shape(heads, m, n, d, dv, &s)) return 0;
  return round256(2ull * heads * n * s.dp * 4) + round256(2ull * heads * s.dvt * s.np * 4) +
         round256(4ull * heads * flag_blocks_of(s.np)) + round256(2ull * kNumSMs * 128 * s.dvp * 4) +
         round256(32ull * heads * s.parts * ((m + 127) / 128));
}

extern "C" int iex_attention_f32(int heads, int m, int n, int d, int dv, const void* plan, const int32_t* row_offsets,
                                 const int32_t* column_indices, const float* q, const float* k, const float* v, float* out,
                                 void* workspace, size_t workspace_bytes, void* stream) {
  if (heads < 0 || m < 0 || n < 0 || d < 0 || dv < 0) return IEX_ERR_BAD_ARG;
  if (heads == 0 || m == 0 || dv == 0) return IEX_OK;
  Shape s;
  if (!attention_shape(heads, m, n, d, dv, &s)) return IEX_ERR_UNSUPPORTED;
  if (!plan || !row_offsets || !column_indices || !q || !k || !v || !out || !workspace) return IEX_ERR_BAD_ARG;
  if (workspace_bytes < iex_attention_workspace_bytes(heads, m, n, d, dv)) return IEX_ERR_TOO_LARGE;
  if (!aligned16(q) || !aligned16(k) || !aligned16(v) || !aligned16(out) || (reinterpret_cast<uintptr_t>(workspace) & 255u))
    return IEX_ERR_UNSUPPORTED;
  uint8_t* ws = static_cast<uint8_t*>(workspace);
  float* k_planes = reinterpret_cast<float*>(ws);
  float* v_planes = reinterpret_cast<float*>(ws + round256(2ull * heads * n * s.dp * 4));
  int* flags = reinterpret_cast<int*>(reinterpret_cast<uint8_t*>(v_planes) + round256(2ull * heads * s.dvt * s.np * 4));
  uint8_t* after = reinterpret_cast<uint8_t*>(flags) + round256(4ull * heads * flag_blocks_of(s.np));
  AttnParams p{};
  p.partials = reinterpret_cast<float4*>(after);
  p.counters = reinterpret_cast<int*>(after + round256(2ull * kNumSMs * 128 * s.dvp * 4));
  p.heads = heads; p.m = m; p.n = n; p.d = d; p.dv = dv;
  p.parts = s.parts;
  p.dvt = s.dvt;
  p.bands = (m + 127) / 128;
  p.tiles = (n + s.kt - 1) / s.kt;
  p.mp = s.mp;
  p.np = s.np;
  p.total = heads * s.parts * p.bands * p.tiles;
  p.bits = static_cast<const uint32_t*>(plan) + 64;
  p.q = q; p.k = k; p.v = v; p.out = out;
  p.row_offsets = row_offsets;
  p.cols = column_indices;
  p.flags = flags;
  p.flag_blocks = flag_blocks_of(s.np);
  p.status = status_word();
  const int sms = std::min(sm_count(), kNumSMs), ctas = cta_count(heads * s.parts * p.bands, p.tiles, sms);
  CUtensorMap mk, mv;
  int st = make_map_f32(&mk, k_planes, 2ll * heads * n, s.dp, s.kt);
  if (st == IEX_OK) st = make_map_f32(&mv, v_planes, 2ll * heads * s.dvt, s.np, s.dvp);
  if (st != IEX_OK) return st;
  cudaStream_t cs = static_cast<cudaStream_t>(stream);
  // The prepare kernel of a call usually follows the main kernel of the one before.  Launched ahead of that kernel's end its
  // blocks would crowd on the few SMs that are free (6 heads x 1003, d 80: 42 us a call instead of 31), so that is
  // done only where main kernels leave a third of the chip free (then it saves 1 to 2 us).
  const dim3 prep_grid(p.flag_blocks, heads + 1);
  const size_t prep_smem = static_cast<size_t>(kPrepKeys) * (dv + 1) * 4;
  if (3 * ctas <= 2 * sms) {
    st = launch_overlapped(attention_prepare_kernel, prep_grid, dim3(256), prep_smem, cs, p, s.dp, k_planes, v_planes, flags);
  } else {
    attention_prepare_kernel<<<prep_grid, 256, prep_smem, cs>>>(p, s.dp, k_planes, v_planes, flags);
    st = launch_status();
  }
  if (st != 0) return st;
  const int which = s.da * 10 + s.dvp / 16;
  switch (which) {
    case 12: return launch_attention<1, 64, 2>(mk, mv, p, ctas, cs);
    case 14: return launch_attention<1, 64, 4>(mk, mv, p, ctas, cs);
    case 22: return launch_attention<2, 64, 2>(mk, mv, p, ctas, cs);
    case 24: return launch_attention<2, 64, 4>(mk, mv, p, ctas, cs);
    case 32: return launch_attention<3, 32, 2>(mk, mv, p, ctas, cs);
    case 34: return launch_attention<3, 32, 4>(mk, mv, p, ctas, cs);
    case 36: return launch_attention<3, 32, 6>(mk, mv, p, ctas, cs);
    case 42: return launch_attention<4, 32, 2>(mk, mv, p, ctas, cs);
    case 44: return launch_attention<4, 32, 4>(mk, mv, p, ctas, cs);
    default: return IEX_ERR_UNSUPPORTED;
  }
}
