// The SDDMM -> SpMM chain of masked attention in one launch over all heads, fp32 in and out:
//   out[h, i, :] = sum over the mask's positions (i, j) of dot(q[h, i], k[h, j]) * v[h, j, :]
//
// Called operator by operator the chain takes a tensor-core SDDMM and a CUDA-core SpMM per head (18 + 22 us
// at 4096 x 4096, 5 %, d = 64; 30 us a head over two streams) plus a few launches' host time per head: the
// SpMM is bound by gathering a row of v per position through L2.  Here both products are dense tiles on
// the tensor cores and the mask is applied in between, in tensor memory, flash-attention style: scores
// never leave the SM and v is read once per 128 rows.
//
// fp32 accuracy: operands are split into fp16 head and tail (x = hi + lo, 22 bits) and three of the four products are kept,
// at twice the rate of the TF32 planes that an earlier version used and with the same number of bits.  What fp16 lacks is
// range, so everything is scaled by powers of two, exactly: a row of q or k to a largest magnitude in [8, 16) (then |S| <
// 2^15 for up to 128 columns), v by the factor its key's row of k lost and by one of its tile (64 or 128 keys), both given
// back when a tile of O is added up.  Tails are stored 2^11 times as large, so that they run out of exponents no sooner than
// the heads; the first head * head instruction scales what the tails' products have summed up back (scale-input-d).  In
// normally distributed data the result is 2.0e-7 off (2-norm), the TF32 planes gave 2.6e-7.
// What leaves fp16's normal range all the same, 2^-14, is held to 2^-36 instead of 2^-22 of itself.  Rows of the mask that this
// could show in are summed position by position at the end (sum_again):
//   v        rows that store a key with such elements (2^-15: 2^-20 of them), or with values that are not finite; in normally
//            distributed data one element in 170 million
//   q and k  rows with a score whose terms' magnitudes sum up to next to nothing: a feature that is large in q and small or zero in
//            k hides what the others give.  That a row of q or k has small elements says too little (normally distributed:
//            one row in 1500), so 32 rows and a tile of keys are compared as a whole first: columns that are large in all of
//            them bound the terms from below (unsafe).  Normally distributed data passes that.
//   factors  rows with a tile whose factor is out of fp32's range (q, k and v of 2^-45 all together, say, or v of 2^110 at one key):
//            its product with the tile's sums need not be.  Tiles say whether some row of q can have one; only then the rows' exponents
//            are looked at (24 heads x 4096, d 64 the same; 6 x 1003, d 80 22.9 -> 24.1 to 24.5 us, as with a branch where a
//            tile is added up; 6 x 1003, d 64 and 128 the same: launches back to back start 1 us apart or a multiple of it).
// The tensor core truncates when it adds to an accumulator, which would bias a sum over thousands of positions (2e-6 of the
// result, measured); a tile's keys are therefore added to fp32 registers with ordinary rounding before the next tile.
//
//   prepare kernel   k and v as hi / lo planes that TMA can load; marks the keys that do not suit and clears the counters
//                    of the bands' pieces (24 heads x 4096 x 64: 100 MB, 23 us cold)
//   main kernel      one persistent CTA per SM over a contiguous run of (head, 128-row band, key tile)
//     warp 0         TMA producer: k and v planes of the next key tiles, q's rows of the next band
//     warp 1         issues S(t) = Q K(t)^T, warp 2 O(t) = P(t) V(t); A operands (Q, P) in tensor memory.  A thread that
//                    issues for a busy tensor pipe pays 200-300 cycles for every barrier it waits on, completed or not, and
//                    70 for a commit.  So there are two of them, each waits once a tile (the barrier of K(t) also counts
//                    the PV that used up the score tile, that of V(t) the warps that wrote P), and a tile has 128 keys where
//                    they fit (1536 cycles of the pipe; with 64 and separate barriers: 313 us instead of 288)
//     warp 3         finds the quarters of a band that may have rows to be summed by position
//     warps 4-11     read S, keep the mask's positions, write P hi / lo over it; add the O of the tile before to
//                    registers.  Two warps per tensor-memory quarter share a tile's columns: the tensor pipe has little else
//                    to do until P(t) is there.  Four per quarter: 294 us, short sequences 25.1 instead of 23.2 us.
//                    They also convert q, from shared memory, under the last PV of the band before (each thread loading its
//                    row from global memory took 7500 cycles a band).
// The runs are equal shares of all tiles; with fewer bands than SMs, every band is cut into the same number of equal pieces
// instead (cta_count).  The pieces of a band meet in a workspace and are added in order by whichever comes last.
//
// 24 heads x 4096 x 4096 at 5 %, d 64: 281 us back to back at the power limit (1590 MHz), about 245 on a cool chip (1965 MHz); with
// TF32 planes 532 to 554 and 499; head by head over two streams 723 us.  About 2260 cycles a tile of 128 keys, of which the
// pipe needs 1536 (68 % active).  From one clock to the other cycles grow by a tenth: memory and the chain S - P - O count too.  6 heads x 1003 x 1003 at 10 %, d 80: 22.6 to 23.3 us, with TF32 planes
// 30.7.  Without a look at the columns of q and k 280 and 22.5.
// Which masks are faster one way or the other: iex_attention_f32_prefers below.
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
int make_map_f16(CUtensorMap* map, const void* base, long long rows, long long cols, long long ld, int box_rows,
                 int box_cols, bool swizzle);  // tc_fused.cu

namespace {

constexpr int kGroups = 2;         // warps that share a quarter of tensor memory: keys and output columns are split between them
constexpr int kThreads = 128 + 128 * kGroups;
constexpr int kMaxTiles = 4;       // tiles at a time: in shared memory and, as scores, in tensor memory
constexpr int kBars = 4 * kMaxTiles + 6;
constexpr int kBarBytes = 8 * kBars + 8;
constexpr int kExpBytes = kGroups * 128;  // exponents of the parts of a band's rows of q
constexpr int kShareBytes = kExpBytes + 4 * 4 * 4 + 3 * 4;  // what quarters of a band have in common; quarters to be looked at
constexpr int kBudget = (227 * 1024 - 1024 - kBarBytes) & ~1023;
constexpr int kRing = kBudget - ((kShareBytes + 1023) & ~1023);  // for the rings and q

constexpr int kTail = 11;      // tails are stored 2^11 times as large: their exponents are then those of the heads
constexpr int kRowExp = 3;     // rows of q and k are scaled to a largest magnitude in [2^3, 2^4): scores stay below 2^15
constexpr int kTileExp = 14;   // a tile of v to [2^14, 2^15)
// Scaled elements of v from here on keep all but 2^-20 of themselves: a tail is 2^-36 off at most where it has no more
// exponents, and as much is lost with the product of the tails.
constexpr float kSmallV = 1.f / (1 << 15);
// Elements of q and k, scaled: a large one; a big one, where one in both rows is enough (sum_again); and from where on fp16 holds them with
// all their bits.
constexpr float kLarge = 1.f / 32, kBig = 1.f / 2, kSmall = 1.f / (1 << 14);
constexpr int kExpBias = 4096;

struct AttnParams {
  int heads, m, n, d, dv;
  int bands, tiles, mp;          // 128-row bands, key tiles of a head, rows of the mask words
  int np, words;                 // keys of a head in the planes (whole tiles), mask words of a row
  int total;                     // heads * bands * tiles
  const uint32_t* bits;          // [key words][mp]
  const float* q;
  const float* k;
  const float* v;
  float* out;
  const int* row_offsets;
  const int* cols;
  float4* partials;              // [2 * CTAs][dvp / 4][128]: sums of a CTA's first and last band where they are cut
  int* counters;                 // [bands of all heads][4 * kGroups]: pieces of a band that are there, per warp ...
  uint32_t* quarters;            // [bands of all heads], 4 bits each: quarters that may have rows to be summed by position; those of a
                                 // band that is cut of which half of the columns is complete; those with pairs that have to be looked
                                 // at; those with rows and tiles whose factor is out of range
  uint32_t* odd_rows;            // [bands of all heads][4]: rows of a quarter that have to be summed by position
  const uint4* tile_info;        // [heads][tiles]: Tile
  const uint32_t* odd_keys;      // [heads][np / 32]: keys that do not suit the planes
  uint4* key_words;              // [heads][np]: big_and_there of the keys of tiles whose info says so
  int* status;
};

__device__ __forceinline__ int range_begin(int c, int total, int ctas) {
  return static_cast<int>(static_cast<long long>(c) * total / ctas);
}

// The CTA whose range holds tile t.
__device__ __forceinline__ int cta_of(int t, int total, int ctas) {
  return static_cast<int>(((t + 1ll) * ctas - 1) / total);
}

// floor(log2 |x|) from the bits of |x| (not 0, finite)
__device__ __forceinline__ int exponent_of(uint32_t bits) {
  return bits >= 0x00800000u ? static_cast<int>(bits >> 23) - 127 : -118 - __clz(bits);
}
// 2^e; 0 below the smallest subnormal, 2^127 above it
__device__ __forceinline__ float power_of_two(int e) {
  if (e >= -126) return __uint_as_float(static_cast<uint32_t>(min(e, 127) + 127) << 23);
  return e < -149 ? 0.f : __uint_as_float(1u << (149 + e));
}
// x * 2^e, in two steps since 2^e alone may be out of range
struct Scale {
  float a, b;
  __device__ __forceinline__ explicit Scale(int e) {
    e = max(-250, min(250, e));
    a = power_of_two(e >> 1);
    b = power_of_two(e - (e >> 1));
  }
  __device__ __forceinline__ float operator()(float x) const { return x * a * b; }
};
// The largest |x| of the finite ones, as bits
__device__ __forceinline__ uint32_t finite_max(uint32_t so_far, float x) {
  const uint32_t b = __float_as_uint(x) & 0x7fffffffu;
  return b < 0x7f800000u ? max(so_far, b) : so_far;
}
// Two numbers as fp16 heads and tails, the tails times 2^11
__device__ __forceinline__ void split2(float2 x, uint32_t& hi, uint32_t& lo) {
  const __half2 h = __floats2half2_rn(x.x, x.y);
  constexpr float kUp = static_cast<float>(1 << kTail);
  float2 t = __fmul2_rn(x, make_float2(kUp, kUp));
  // x * 2^11 - h * 2^11 straight from the fp16 numbers
  asm("{\n\t.reg .b16 a, b, c;\n\tmov.b32 {a, b}, %2;\n\tmov.b16 c, %3;\n\t"
      "fma.rn.f32.f16 %0, a, c, %0;\n\tfma.rn.f32.f16 %1, b, c, %1;\n\t}"
      : "+f"(t.x), "+f"(t.y)
      : "r"(*reinterpret_cast<const uint32_t*>(&h)), "n"(0xe800));  // -2^11
  const __half2 l = __floats2half2_rn(t.x, t.y);
  hi = *reinterpret_cast<const uint32_t*>(&h);
  lo = *reinterpret_cast<const uint32_t*>(&l);
}

// A key tile as its prepare block describes it: v's rows times k's scales are stored times 2^-exponent; whether keys of it do not
// suit the planes; the most small elements that a key's row of k has; the columns that are large in all of them; whether its keys'
// words are in key_words.  Of the first 64
// columns c is bit (c % 32) / 2 of word c / 32, odd ones 16 further.  A key whose row is zero counts for neither.
struct Tile {
  uint32_t word, large0, large1;
  __device__ __forceinline__ explicit Tile(const uint4* at) {
    const uint4 x = __ldcg(at);
    word = x.x;
    large0 = x.y;
    large1 = x.z;
  }
  static __device__ __forceinline__ uint4 pack(int exponent, bool odd, int small, uint32_t large0, uint32_t large1, bool described) {
    return make_uint4(static_cast<uint32_t>(exponent + kExpBias) | (odd ? 1u << 13 : 0u) | static_cast<uint32_t>(small) << 14, large0,
                      large1, described ? 1u : 0u);
  }
  static __device__ __forceinline__ int exponent(uint32_t word) { return static_cast<int>(word & 0x1fffu) - kExpBias; }
  __device__ __forceinline__ bool odd() const { return (word & (1u << 13)) != 0; }
  __device__ __forceinline__ int small() const { return static_cast<int>(word >> 14); }
};
// Whether scores of some rows of q and a tile's keys can be off by more than 2^-21 of their terms, or P, which follows from them.
// Of the first 64 columns `large` are large in all these rows but the zero ones, and a row of q and a key together have at most
// `small` small elements (zeros too, which is on the safe side).  A small element is 2^-36 off and as much is lost with the product
// of the tails, times at most 16 from the other side: 2^-31.  A large column adds 2^-10 or more to the terms, so that with a small
// element for each of them 2^-21 of the terms is lost; and P, 2^-35 off at most, wants the terms to be 2^-14.
__device__ __forceinline__ bool unsafe(int large, int small) { return large == 0 || small > large; }
// Whether 2^exponent, the factor of a tile's sums O, is no fp32 number.  O is up to 2^37 and may be small, so O * 2^exponent can be one.
__device__ __forceinline__ bool out_of_range(int exponent) { return exponent < -149 || exponent > 127; }
// The same for some row of q, whose share is in [-126, 127] - 2 kRowExp.
__device__ __forceinline__ bool may_be_out_of_range(int tile_exponent) {
  return out_of_range(tile_exponent - 126 - 2 * kRowExp) || out_of_range(tile_exponent + 127 - 2 * kRowExp);
}

__device__ __forceinline__ void umma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc,
                                            uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem_d),
      "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// D = A B + D * 2^-kTail
__device__ __forceinline__ void umma_f16_ts_scaled(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.eq.b32 p, 0, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p, %4;\n\t}" ::"r"(tmem_d),
      "r"(tmem_a), "l"(bdesc), "r"(idesc), "n"(kTail)
      : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t* r) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(r[0]),
               "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
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
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// Words of a row of q or k, scaled, for pairs of rows: columns of the first 64 that are big, and those that are not zero, c beside
// c + 64 (a row's 16 threads have 4 columns each, or twice 4; two rows a warp).
__device__ __forceinline__ uint4 big_and_there(const float4& a, const float4& b) {
  const int shift = threadIdx.x & 16;
  auto word = [&](bool even, bool odd) -> uint32_t {
    return (__ballot_sync(0xffffffffu, even) >> shift & 0xffffu) | __ballot_sync(0xffffffffu, odd) >> shift << 16;
  };
  const uint32_t big0 = word(fabsf(a.x) >= kBig, fabsf(a.y) >= kBig), big1 = word(fabsf(a.z) >= kBig, fabsf(a.w) >= kBig);
  return make_uint4(big0, big1, word(a.x != 0.f || b.x != 0.f, a.y != 0.f || b.y != 0.f),
                    word(a.z != 0.f || b.z != 0.f, a.w != 0.f || b.w != 0.f));
}
__device__ __forceinline__ float4 scaled4(const Scale& s, const float4& x) { return make_float4(s(x.x), s(x.y), s(x.z), s(x.w)); }

// big_and_there of rows [0, rows) of q or k at `x` into `to`, by all threads of the block, 8 rows on their way for each; no exponent
// below `lowest`.
__device__ __forceinline__ void row_words(const float* x, int rows, int d, int lowest, uint4* to) {
  constexpr int kRows = 8, kSide = kThreads / 16;
  const int lane16 = threadIdx.x & 15;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int row0 = 0; row0 < rows; row0 += kRows * kSide) {
    float4 a[kRows], b[kRows];
#pragma unroll
    for (int i = 0; i < kRows; ++i) {
      const int row = row0 + i * kSide + static_cast<int>(threadIdx.x >> 4);
      const float4* from = reinterpret_cast<const float4*>(x + static_cast<size_t>(row) * d);
      a[i] = row < rows && 4 * lane16 < d ? __ldg(from + lane16) : zero;
      b[i] = row < rows && 64 + 4 * lane16 < d ? __ldg(from + 16 + lane16) : zero;
    }
#pragma unroll
    for (int i = 0; i < kRows; ++i) {
      const int row = row0 + i * kSide + static_cast<int>(threadIdx.x >> 4);
      uint32_t top = finite_max(finite_max(finite_max(finite_max(0u, a[i].x), a[i].y), a[i].z), a[i].w);
      top = finite_max(finite_max(finite_max(finite_max(top, b[i].x), b[i].y), b[i].z), b[i].w);
#pragma unroll
      for (int s = 8; s >= 1; s >>= 1) top = max(top, __shfl_xor_sync(0xffffffffu, top, s));
      const Scale scale(top != 0u ? kRowExp - max(exponent_of(top), lowest) : 0);
      const uint4 words = big_and_there(scaled4(scale, a[i]), scaled4(scale, b[i]));
      if (lane16 == 0 && row < rows) to[row] = words;
    }
  }
}

// By a warp: whether a row of q and a key have terms in common and these are next to nothing: below 2^-14 or, with small elements, below
// what makes 2^-31 for each of them 2^-21.
__device__ __noinline__ bool next_to_nothing(const float4* q, const float4* k, int quads) {
  const int lane = threadIdx.x & 31;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f), a = lane < quads ? __ldg(q + lane) : zero, b = lane < quads ? __ldg(k + lane) : zero;
  const uint32_t top_q = __reduce_max_sync(0xffffffffu, finite_max(finite_max(finite_max(finite_max(0u, a.x), a.y), a.z), a.w));
  const uint32_t top_k = __reduce_max_sync(0xffffffffu, finite_max(finite_max(finite_max(finite_max(0u, b.x), b.y), b.z), b.w));
  if (top_q == 0u || top_k == 0u) return false;
  const Scale scale_q(kRowExp - max(exponent_of(top_q), -126)), scale_k(kRowExp - exponent_of(top_k));
  float terms = 0.f;
  int small = 0;
  bool any = false;
  auto add = [&](float u, float v) {
    const float x = fabsf(scale_q(u)), y = fabsf(scale_k(v));
    any = any || (u != 0.f && v != 0.f);
    small += (u != 0.f && x < kSmall ? 1 : 0) + (v != 0.f && y < kSmall ? 1 : 0);
    terms = fmaf(x, y, terms);
  };
  add(a.x, b.x);
  add(a.y, b.y);
  add(a.z, b.z);
  add(a.w, b.w);
#pragma unroll
  for (int w = 16; w >= 1; w >>= 1) terms += __shfl_xor_sync(0xffffffffu, terms, w);
  small = __reduce_add_sync(0xffffffffu, small);
  return __any_sync(0xffffffffu, any) && terms < fmaxf(kSmall, small * (1.f / 1024));
}

// Quarters of a band that have rows and tiles [0, tiles) whose factor is out of range, from the exponent bytes of the rows (a warp).
__device__ __noinline__ uint32_t far_quarters(const volatile uint8_t* exps, int rows, const uint4* info, int tiles) {
  const int lane = threadIdx.x & 31;
  int lowest = 10000, highest = -10000;
  for (int t = lane; t < tiles; t += 32) {
    const int e = Tile::exponent(__ldcg(&info[t].x));
    lowest = min(lowest, e);
    highest = max(highest, e);
  }
  lowest = __reduce_min_sync(0xffffffffu, lowest);
  highest = __reduce_max_sync(0xffffffffu, highest);
  uint32_t far = 0;
#pragma unroll 1
  for (int i = 0; i < 4; ++i) {
    const int row = 32 * i + lane;
    int e = 0;
    for (int w = 0; w < kGroups; ++w) e = max(e, static_cast<int>(exps[w * 128 + row]));
    e -= 127 + 2 * kRowExp;
    if (__any_sync(0xffffffffu, e != -127 - 2 * kRowExp && row < rows && (out_of_range(e + lowest) || out_of_range(e + highest))))
      far |= 1u << i;
  }
  return far;
}

// Marks the rows of a quarter of a band (a warp) that have a tile whose factor is out of range.
__device__ __noinline__ void mark_far(const AttnParams& p, int item, int part) {
  const int head = item / p.bands, lane = threadIdx.x & 31, row = (item - head * p.bands) * 128 + part * 32 + lane;
  const float4* q = reinterpret_cast<const float4*>(p.q + (static_cast<size_t>(head) * p.m + min(row, p.m - 1)) * p.d);
  const uint4* info = p.tile_info + head * p.tiles;
  uint32_t top = 0;
#pragma unroll 1
  for (int c = 0; c < p.d / 4; ++c) {
    const float4 a = __ldg(q + c);
    top = finite_max(finite_max(finite_max(finite_max(top, a.x), a.y), a.z), a.w);
  }
  bool far = false;
  const int e = max(exponent_of(max(top, 1u)), -126) - 2 * kRowExp;
#pragma unroll 1
  for (int t = 0; t < p.tiles; ++t) far = far || out_of_range(e + Tile::exponent(__ldcg(&info[t].x)));
  const uint32_t rows = __ballot_sync(0xffffffffu, far && top != 0u && row < p.m);
  if (lane == 0 && rows != 0) atomicOr(p.odd_rows + 4 * item + part, rows);
}

// Row r of a head position by position (a warp), 32 at a time: 8 lanes share a score, and a row of v takes a lane for 4 columns, two
// rows at a time up to 64 columns.
__device__ __forceinline__ void row_by_position(const AttnParams& p, int head, int r, int lane) {
  const float* k = p.k + static_cast<size_t>(head) * p.n * p.d;
  const float* v = p.v + static_cast<size_t>(head) * p.n * p.dv;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  const int lane8 = lane & 7, split = p.dv <= 64 ? 2 : 1, half = split == 2 ? lane >> 4 : 0;
  const int vc = split == 2 ? lane & 15 : lane;  // this lane's 4 columns of v
  auto add = [](float4& to, const float4& a, const float4& b) {
    to.x = fmaf(a.x, b.x, to.x);
    to.y = fmaf(a.y, b.y, to.y);
    to.z = fmaf(a.z, b.z, to.z);
    to.w = fmaf(a.w, b.w, to.w);
  };
  const int begin = __ldg(p.row_offsets + r), end = __ldg(p.row_offsets + r + 1);
  const float4* q = reinterpret_cast<const float4*>(p.q + (static_cast<size_t>(head) * p.m + r) * p.d);
  float4 q4[4], acc = zero;
#pragma unroll
  for (int c = 0; c < 4; ++c) q4[c] = lane8 + 8 * c < p.d / 4 ? __ldg(q + lane8 + 8 * c) : zero;
  int coming = begin + lane < end ? __ldg(p.cols + begin + lane) : 0;
  for (int e = begin; e < end; e += 32) {
    const int j = coming, here = min(32, end - e);
    coming = e + 32 + lane < end ? __ldg(p.cols + e + 32 + lane) : 0;
    float score = 0.f;  // of position e + lane
#pragma unroll
    for (int u0 = 0; u0 < 8; u0 += 4) {
      float4 x[4][4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int key = __shfl_sync(0xffffffffu, j, 4 * (u0 + u) + (lane >> 3));  // key 0 past the end
        const float4* kj = reinterpret_cast<const float4*>(k + static_cast<size_t>(key) * p.d);
#pragma unroll
        for (int c = 0; c < 4; ++c) x[u][c] = lane8 + 8 * c < p.d / 4 ? __ldg(kj + lane8 + 8 * c) : zero;
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        float4 part = zero;
#pragma unroll
        for (int c = 0; c < 4; ++c)
          if (lane8 + 8 * c < p.d / 4) add(part, q4[c], x[u][c]);
        float s = (part.x + part.y) + (part.z + part.w);
#pragma unroll
        for (int w = 4; w >= 1; w >>= 1) s += __shfl_xor_sync(0xffffffffu, s, w);
        // position 4 (u0 + u) + i is in lanes 8 i to 8 i + 7
        const float mine = __shfl_sync(0xffffffffu, s, 8 * (lane & 3));
        if (lane >> 2 == u0 + u) score = mine;
      }
    }
#pragma unroll 1
    for (int u0 = 0; u0 < here; u0 += 16 * split) {
      float4 x[16];
#pragma unroll
      for (int u = 0; u < 16; ++u) {
        const int key = __shfl_sync(0xffffffffu, j, (u0 + split * u + half) & 31);
        x[u] = 4 * vc < p.dv ? __ldg(reinterpret_cast<const float4*>(v + static_cast<size_t>(key) * p.dv) + vc) : zero;
      }
#pragma unroll
      for (int u = 0; u < 16; ++u) {
        const int at = u0 + split * u + half;
        const float f = __shfl_sync(0xffffffffu, score, at & 31);
        if (at < here) add(acc, make_float4(f, f, f, f), x[u]);
      }
    }
  }
  if (split == 2) {
    acc.x += __shfl_down_sync(0xffffffffu, acc.x, 16);
    acc.y += __shfl_down_sync(0xffffffffu, acc.y, 16);
    acc.z += __shfl_down_sync(0xffffffffu, acc.z, 16);
    acc.w += __shfl_down_sync(0xffffffffu, acc.w, 16);
  }
  if (half == 0 && 4 * vc < p.dv) reinterpret_cast<float4*>(p.out + (static_cast<size_t>(head) * p.m + r) * p.dv)[vc] = acc;
}

// After everything else, by all threads: rows of this block's bands, tiles [r0, r1), that have to be summed by position.  `cut`:
// the quarters (4 bits each) of its first and its last band that it has to see to where these are cut between blocks; all others,
// and whether there may be such rows in them, are in p.quarters.  Which rows that are is found from the words of q's and k's rows: a
// column that is big on both sides makes a pair's terms 1 / 4 or more, enough for 256 small elements, and nothing in common makes them
// zero; other pairs are looked at.  `words`: shared memory for kAgainWords of them.
// 24 heads x 4096, d 64 on a cool chip (245 us otherwise): one key in every head 415 us, q and k after a ReLU, where all pairs are
// looked at, 440, one column of q and k 2^4 times the others 465, 2^8 times 610, and one of q 2^24, one of k 2^-24 times the others,
// where every row is summed, 2200.  (A lane for a pair and big only from 1 on: 710, 1080 and 2980 for the last three.)  At the end
// and not in the loop over the tiles: any code there that looks at the scores, even if it is
// passed over, makes the loop 3 to 12 % longer, and so does one that keeps such a row's number.
constexpr int kAgainKeys = 8192, kAgainWords = kAgainKeys + 128;
__device__ __noinline__ void sum_again(const AttnParams& p, int r0, int r1, uint32_t cut, uint4* words) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, part = warp & 3;
  struct Band {
    int item, head, row0, rows;
    uint32_t quarters, pairs, far;  // to look at; with pairs to be looked at; with rows that may have factors out of range
  };
  auto band_of = [&](int r) -> Band {
    const int item = r / p.tiles, head = item / p.bands, row0 = (item - head * p.bands) * 128, first = item * p.tiles;
    const uint32_t marks = __ldcg(p.quarters + item);
    const uint32_t mine = r == first && r1 - first >= p.tiles ? 15u : (r == r0 ? cut : cut >> 4) & 15u;
    return {item, head, row0, min(128, p.m - row0), marks & mine, marks >> 8 & mine, marks >> 12 & mine};
  };
  auto next_band = [&](int r) { return (r / p.tiles + 1) * p.tiles; };
  uint4* q_words = words + kAgainKeys;
  int held = -1;  // head whose keys' words are there
  for (int r = r0; r < r1; r = next_band(r)) {
    const Band at = band_of(r);
    if (at.quarters == 0) continue;
    if (warp < 4 && at.far >> part & 1u) mark_far(p, at.item, part);
    __syncthreads();
    if (at.pairs != 0) row_words(p.q + (static_cast<size_t>(at.head) * p.m + at.row0) * p.d, at.rows, p.d, -126, q_words);
    for (int key0 = 0; key0 < p.n; key0 += kAgainKeys) {
      const int keys = min(kAgainKeys, p.n - key0);
      __syncthreads();
      if (at.pairs != 0 && (held != at.head || keys != p.n)) {
        const uint4* info = p.tile_info + at.head * p.tiles;
        bool described = true;
        for (int t = threadIdx.x; t < p.tiles; t += kThreads) described = described && __ldcg(&info[t].w) != 0u;
        if (__syncthreads_and(described)) {
          const uint4* from = p.key_words + static_cast<size_t>(at.head) * p.np + key0;
          for (int i = threadIdx.x; i < keys; i += kThreads) words[i] = __ldcg(from + i);
        } else {
          row_words(p.k + (static_cast<size_t>(at.head) * p.n + key0) * p.d, keys, p.d, -149, words);
        }
        held = at.head;
      }
      __syncthreads();
      if (!(at.quarters >> part & 1u)) continue;
      // a warp takes every third run of 32 words of mask of a quarter
      const bool pairs = at.pairs >> part & 1u;
      const int row = part * 32 + lane;
      const uint4 mine = row < at.rows && pairs ? q_words[row] : make_uint4(0u, 0u, 0u, 0u);
      const uint32_t* mask = p.bits + static_cast<size_t>(key0 / 32) * p.mp + at.row0 + row;
      const uint32_t* odd_keys = p.odd_keys + (static_cast<size_t>(at.head) * p.np + key0) / 32;
      const int count = (keys + 31) / 32;
      bool found = row >= at.rows;
      for (int w0 = warp >> 2; w0 < count; w0 += 32 * (kThreads / 128)) {
        const int mine_at = w0 + lane * (kThreads / 128);
        const uint32_t odd_here = mine_at < count ? __ldcg(odd_keys + mine_at) : 0u;
        const uint32_t visit = pairs ? 0xffffffffu : __ballot_sync(0xffffffffu, odd_here != 0);
        auto bits_of = [&](int i) -> uint32_t {
          const int w = w0 + i * (kThreads / 128);
          return i < 32 && w < count && !found && visit >> i & 1u ? __ldg(mask + static_cast<size_t>(w) * p.mp) : 0u;
        };
        uint32_t coming = bits_of(0);
        for (int i = 0; i < 32 && w0 + i * (kThreads / 128) < count; ++i) {
          uint32_t bits = coming;
          coming = bits_of(i + 1);
          const uint32_t odd = __shfl_sync(0xffffffffu, odd_here, i);  // by all lanes, found or not
          found = found || (bits & odd) != 0;
          if (!pairs) continue;
          for (;;) {  // pairs that the words leave open, one of each row at a time, are looked at by the warp
            int key = -1;
            for (; bits != 0 && !found && key < 0; bits &= bits - 1) {
              const int next = 32 * (w0 + i * (kThreads / 128)) + __ffs(bits) - 1;
              const uint4 theirs = words[next];
              if (((mine.x & theirs.x) | (mine.y & theirs.y)) == 0 && ((mine.z & theirs.z) | (mine.w & theirs.w)) != 0) key = next;
            }
            uint32_t open = __ballot_sync(0xffffffffu, key >= 0);
            if (open == 0) break;
            for (; open != 0; open &= open - 1) {
              const int whose = __ffs(open) - 1, which = __shfl_sync(0xffffffffu, key, whose);
              const float* q = p.q + (static_cast<size_t>(at.head) * p.m + at.row0 + part * 32 + whose) * p.d;
              const float* k = p.k + (static_cast<size_t>(at.head) * p.n + key0 + which) * p.d;
              const bool next_to = next_to_nothing(reinterpret_cast<const float4*>(q), reinterpret_cast<const float4*>(k), p.d / 4);
              found = found || (lane == whose && next_to);
            }
          }
        }
      }
      const uint32_t odd = __ballot_sync(0xffffffffu, found && row < at.rows);
      if (lane == 0 && odd != 0) atomicOr(p.odd_rows + 4 * at.item + part, odd);
    }
  }
  __threadfence();
  __syncthreads();
  int turn = 0;  // the warps take the rows in turn
  for (int r = r0; r < r1; r = next_band(r)) {
    const Band at = band_of(r);
    for (int i = 0; i < 4; ++i)
      for (uint32_t odd = at.quarters >> i & 1u ? __ldcg(p.odd_rows + 4 * at.item + i) : 0u; odd != 0; odd &= odd - 1) {
        if (turn == warp) row_by_position(p, at.head, at.row0 + i * 32 + __ffs(odd) - 1, lane);
        if (++turn == kThreads / 32) turn = 0;
      }
  }
}

// kQ: columns of q and k (d rounded up to 64 or 128), KT: keys per tile, DVP: columns of v (dv rounded up)
template <int kQ, int KT, int DVP>
struct Layout {
  static constexpr int kKAtoms = kQ / 64, kVAtoms = (DVP + 63) / 64;  // 64 fp16 numbers: one 128-byte swizzle atom
  static constexpr int kKPlane = KT * 128 * kKAtoms, kVPlane = KT * 128 * kVAtoms;
  static constexpr int kQBytes = kQ / 32 * 16384;
  static constexpr int kTensor = (512 - kQ - 2 * DVP) / KT, kShared = (kRing - kQBytes) / (2 * (kKPlane + kVPlane));
  static constexpr int kFit = kTensor < kShared ? kTensor : kShared, kTiles = kFit < kMaxTiles ? kFit : kMaxTiles;
  static_assert(kTiles >= 2, "two tiles at a time");
};

template <int kQ, int KT, int DVP>
__global__ void __launch_bounds__(kThreads, 1)
attention_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                 const __grid_constant__ CUtensorMap map_v, const __grid_constant__ AttnParams p) {
  using L = Layout<kQ, KT, DVP>;
  constexpr int kKAtoms = L::kKAtoms, kVAtoms = L::kVAtoms, kTiles = L::kTiles;
  constexpr uint32_t kKPlane = L::kKPlane, kVPlane = L::kVPlane;
  constexpr uint32_t kQHi = 0, kQLo = kQ / 2, kS = kQ, kO = kQ + kTiles * KT;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* base_ptr = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t bar = base + kBudget;
  // Of tile t, with b = t % kTiles: K(t) is there and P(t - kTiles) used up; S(t); P(t) and V(t) are there; O(t)
  auto k_full = [&](int b) { return bar + 8u * b; };
  auto s_full = [&](int b) { return bar + 8u * (kMaxTiles + b); };
  auto p_full = [&](int b) { return bar + 8u * (2 * kMaxTiles + b); };
  auto pv_done = [&](int b) { return bar + 8u * (3 * kMaxTiles + b); };
  const uint32_t v_base = base + kTiles * 2u * kKPlane, q_base = v_base + kTiles * 2u * kVPlane;
  constexpr uint32_t kB1 = 32u * kMaxTiles;
  const uint32_t q_full = bar + kB1, raw_full = bar + kB1 + 8u, raw_empty = bar + kB1 + 16u, exps_there = bar + kB1 + 24u,
                 looked_at = bar + kB1 + 32u;  // the first band, and 8 further the last one, by warp 3
  volatile uint32_t* tmem_ptr = reinterpret_cast<volatile uint32_t*>(base_ptr + kBudget + 8 * kBars);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_ptr + 1);
  // Of each quarter of a band: columns of the first 64 that are large in all its rows (as in Tile), the most small elements of a
  // row in each of its warps' columns
  volatile uint32_t* common = reinterpret_cast<volatile uint32_t*>(base_ptr + kRing + kExpBytes);
  // quarters that this block has to see to at the end, if there is anything: of its first band, of its last; 256: of others
  uint32_t* again = reinterpret_cast<uint32_t*>(base_ptr + kRing + kExpBytes + 64);
  volatile uint32_t* piece = again + 1;  // quarters of the first band, and of the last, as far as this block's tiles tell

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int b = 0; b < kMaxTiles; ++b) {
      mbar_init(k_full(b), 2);
      mbar_init(s_full(b), 1);
      mbar_init(p_full(b), 4 * kGroups + 1);
      mbar_init(pv_done(b), 1);
    }
    mbar_init(q_full, 4 * kGroups);
    mbar_init(raw_full, 1);
    mbar_init(raw_empty, 4 * kGroups + 1);
    mbar_init(exps_there, 4 * kGroups);
    mbar_init(looked_at, 1);
    mbar_init(looked_at + 8u, 1);
    *abort_flag = 0;
    *again = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    for (int b = 0; b < kTiles; ++b) mbar_arrive(k_full(b));  // nothing to use up before the first tiles
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
      asm volatile("prefetch.tensormap [%0];" ::"l"(&map_q) : "memory");
      asm volatile("prefetch.tensormap [%0];" ::"l"(&map_k) : "memory");
      asm volatile("prefetch.tensormap [%0];" ::"l"(&map_v) : "memory");
      int b = 0;
      uint32_t ph = 0, seg = 0;
      const int q_atoms = (p.d + 31) / 32;
      for (int r = r0; r < r1; ++r) {
        const int item = r / p.tiles, t = r - item * p.tiles, head = item / p.bands;
        if (r == r0 || t == 0) {  // the band's rows of q as they are
          if (!mbar_wait(raw_empty, (seg & 1u) ^ 1u, abort_flag, p.status, 32)) break;
          mbar_arrive_expect_tx(raw_full, q_atoms * 16384u);
          for (int a = 0; a < q_atoms; ++a)
            tma_load_2d(q_base + a * 16384u, &map_q, raw_full, a * 32, head * p.m + (item - head * p.bands) * 128);
          ++seg;
        }
        if (!mbar_wait(s_full(b), ph ^ 1u, abort_flag, p.status, 32)) break;
        mbar_arrive_expect_tx(k_full(b), 2 * kKPlane);
#pragma unroll
        for (int pl = 0; pl < 2; ++pl)
#pragma unroll
          for (int a = 0; a < kKAtoms; ++a)
            tma_load_2d(base + (2 * b + pl) * kKPlane + a * (KT * 128), &map_k, k_full(b), a * 64,
                        (pl * p.heads + head) * p.np + t * KT);
        if (!mbar_wait(pv_done(b), ph ^ 1u, abort_flag, p.status, 32)) break;
        mbar_arrive_expect_tx(p_full(b), 2 * kVPlane);
#pragma unroll
        for (int pl = 0; pl < 2; ++pl)
#pragma unroll
          for (int a = 0; a < kVAtoms; ++a)
            tma_load_2d(v_base + (2 * b + pl) * kVPlane + a * (KT * 128), &map_v, p_full(b), a * 64,
                        (pl * p.heads + head) * p.np + t * KT);
        if (++b == kTiles) { b = 0; ph ^= 1u; }
      }
      if (*abort_flag)
        for (uint32_t i = 0; i < 2048u; ++i) __nanosleep(100);
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------------------ S = Q K^T
    if (elect_one()) {
      constexpr uint32_t idesc = (1u << 4) | (static_cast<uint32_t>(KT >> 3) << 17) | (8u << 24);
      const int steps = (p.d + 15) / 16;
      int b = 0;
      uint32_t ph = 0, seg = 0;
      bool ok = true;
      for (int r = r0; r < r1 && ok; ++seg) {
        const int seg_end = min(r1, (r / p.tiles + 1) * p.tiles);
        if (!mbar_wait(q_full, seg & 1u, abort_flag, p.status, 20)) break;
        for (; r < seg_end; ++r) {
          if (!mbar_wait(k_full(b), ph, abort_flag, p.status, 20)) { ok = false; break; }
          tcgen05_fence_after();
          const uint32_t k_hi = base + 2 * b * kKPlane, d = tmem + kS + b * KT;
          // small terms first: tail * head', head * tail', then, with those scaled back, head * head'
#pragma unroll
          for (int pr = 0; pr < 3; ++pr)
#pragma unroll
            for (int a = 0; a < kKAtoms; ++a) {
              const uint64_t bd = smem_desc(k_hi + (pr == 1 ? kKPlane : 0u) + a * (KT * 128), 16, 1024);
#pragma unroll
              for (int ks = 0; ks < 4; ++ks) {
                if (a * 4 + ks >= steps) continue;
                const uint32_t qa = tmem + (pr == 0 ? kQLo : kQHi) + a * 32 + ks * 8;
                if (pr == 2 && a == 0 && ks == 0) umma_f16_ts_scaled(d, qa, bd, idesc);
                else umma_f16_ts(d, qa, desc_advance(bd, ks * 32), idesc, (pr | a | ks) != 0 ? 1u : 0u);
              }
            }
          umma_commit(s_full(b));
          if (++b == kTiles) { b = 0; ph ^= 1u; }
        }
      }
    }
    __syncwarp();
  } else if (warp == 2) {
    // ------------------------------------------------------------------ O = P V
    if (elect_one()) {
      const uint32_t idesc = (1u << 4) | (1u << 16) | (static_cast<uint32_t>((p.dv + 15) / 16 * 2) << 17) | (8u << 24);
      int b = 0;
      uint32_t ph = 0;
      for (int r = r0; r < r1; ++r) {
        // P(g) also says that O(g - 2) has been read: every warp adds it before it writes P(g)
        if (!mbar_wait(p_full(b), ph, abort_flag, p.status, 20)) break;
        tcgen05_fence_after();
        const uint32_t v_hi = v_base + 2 * b * kVPlane, d = tmem + kO + ((r - r0) & 1) * DVP, pp = tmem + kS + b * KT;
#pragma unroll
        for (int pr = 0; pr < 3; ++pr) {
          const uint64_t bd = smem_desc(v_hi + (pr == 1 ? kVPlane : 0u), KT * 128, 1024);
#pragma unroll
          for (int ks = 0; ks < KT / 16; ++ks) {  // 16 keys of P: 8 columns of heads, 8 of tails
            const uint32_t pa = pp + ks * 16 + (pr == 0 ? 8 : 0);
            if (pr == 2 && ks == 0) umma_f16_ts_scaled(d, pa, bd, idesc);
            else umma_f16_ts(d, pa, desc_advance(bd, ks * (16 * 128)), idesc, (pr | ks) != 0 ? 1u : 0u);
          }
        }
        umma_commit(pv_done(b));
        if (r + kTiles < r1) umma_commit(k_full(b));
        if (++b == kTiles) { b = 0; ph ^= 1u; }
      }
    }
    __syncwarp();
  } else if (warp == 3) {
    // ------------------------------------------------------------------ quarters that may have rows to be summed by position
    uint32_t seg = 0;
    for (int r = r0; r < r1; ++seg) {
      const int item = r / p.tiles, first = item * p.tiles, seg_end = min(r1, first + p.tiles);
      const uint4* info = p.tile_info + item / p.bands * p.tiles;
      if (!mbar_wait(q_full, seg & 1u, abort_flag, p.status, 200)) break;
      __syncwarp();
      const uint32_t mine = common[lane & 15];
      uint32_t quarters = 0;
      bool far = false;
      for (int t = r - first; t < seg_end - first; t += 32) {
        const Tile tile(info + min(t + lane, seg_end - first - 1));
        far = far || may_be_out_of_range(Tile::exponent(tile.word));
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const uint32_t large0 = __shfl_sync(0xffffffffu, mine, 4 * i) & tile.large0;
          const uint32_t large1 = __shfl_sync(0xffffffffu, mine, 4 * i + 1) & tile.large1;
          const int small = static_cast<int>(__shfl_sync(0xffffffffu, mine, 4 * i + 2) + __shfl_sync(0xffffffffu, mine, 4 * i + 3));
          if (tile.odd()) quarters |= 1u << i;
          if (unsafe(__popc(large0) + __popc(large1), small + tile.small())) quarters |= 0x101u << i;
        }
      }
      quarters = __reduce_or_sync(0xffffffffu, quarters);
      if (__any_sync(0xffffffffu, far))
        quarters |= 0x1001u * far_quarters(base_ptr + kRing, p.m - item % p.bands * 128, info + (r - first), seg_end - r);
      __syncwarp();
      if (lane == 0) mbar_arrive(raw_empty);  // the next band's may be written
      if (lane == 0) {
        if (quarters != 0) {
          atomicOr(p.quarters + item, quarters);
          if (seg_end - r == p.tiles) atomicOr(again, 256u);
        }
        if (r == r0 || seg_end == r1) {
          const int which = r == r0 ? 0 : 1;
          piece[which] = quarters;
          mbar_arrive(looked_at + 8u * which);
        }
      }
      r = seg_end;
    }
  } else {
    // ------------------------------------------------------------------ mask and sums
    const int wg = (warp >> 2) - 1, q4 = warp & 3;
    const uint32_t lanes = tmem + (static_cast<uint32_t>(q4 * 32) << 16);
    const int row_local = q4 * 32 + lane;
    // This warp group's share of a band's q columns into tensor memory; the band's sums are those of O times 2^row_exp, and the
    // tile's exponent.
    const uint8_t* q_ptr = base_ptr + (q_base - base);
    volatile uint8_t* exp_ptr = base_ptr + kRing;
    auto put_q = [&](uint32_t seg, int band, int& row_exp) -> bool {
      constexpr int kShare = kQ / kGroups;
      if (!mbar_wait(raw_full, seg & 1u, abort_flag, p.status, 20)) return false;
      // four columns; 128-byte swizzle; whole 32-column atoms are there
      auto quad = [&](int c) -> float4 {
        const float4 x = *reinterpret_cast<const float4*>(q_ptr + (c >> 5) * 16384 + row_local * 128 + ((((c >> 2) & 7) ^ (row_local & 7)) << 4));
        return c < p.d ? x : make_float4(0.f, 0.f, 0.f, 0.f);
      };
      uint32_t top = 0;
#pragma unroll
      for (int h = 0; h < kShare / 16; ++h)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float4 x = quad(wg * kShare + 16 * h + 4 * j);
          top = finite_max(finite_max(finite_max(finite_max(top, x.x), x.y), x.z), x.w);
        }
      exp_ptr[wg * 128 + row_local] = static_cast<uint8_t>(top != 0u ? max(top >> 23, 1u) : 0u);
      __syncwarp();
      if (lane == 0) mbar_arrive(exps_there);
      if (!mbar_wait(exps_there, seg & 1u, abort_flag, p.status, 20)) return false;
      int e = 0;
#pragma unroll
      for (int i = 0; i < kGroups; ++i) e = max(e, static_cast<int>(exp_ptr[i * 128 + row_local]));
      const bool counts = e != 0 && band * 128 + row_local < p.m;
      e = max(e, 1) - 127;  // of the whole row; of subnormal ones as of 2^-126
      const Scale scale(kRowExp - e);
      row_exp = e - 2 * kRowExp;
      uint32_t large = 0, smalls = 0;
#pragma unroll
      for (int h = 0; h < kShare / 16; ++h) {
        if (kQ == 128 && h % 2 == 0 && wg * kShare + 16 * h >= p.d) break;  // nothing multiplies these columns
        uint32_t hi[8], lo[8], large_here = 0, small_here = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float4 f = quad(wg * kShare + 16 * h + 4 * j);
          split2(make_float2(scale(f.x), scale(f.y)), hi[2 * j], lo[2 * j]);
          split2(make_float2(scale(f.z), scale(f.w)), hi[2 * j + 1], lo[2 * j + 1]);
        }
        tmem_st8(lanes + kQHi + wg * (kShare / 2) + h * 8, hi);
        tmem_st8(lanes + kQLo + wg * (kShare / 2) + h * 8, lo);
#pragma unroll
        for (int j = 0; j < 8; ++j) {  // a bit for even columns, 16 further one for odd ones
          const __half2 x = __habs2(*reinterpret_cast<const __half2*>(&hi[j]));
          large_here |= (0x00010001u << j) & __hge2_mask(x, __float2half2_rn(kLarge));
          small_here |= (0x00010001u << j) & __hlt2_mask(x, __float2half2_rn(kSmall));
        }
        const int here = min(max(p.d - (wg * kShare + 16 * h), 0), 16);  // columns that there are
        smalls += __popc(small_here & ((1u << here / 2) - 1u) * 0x00010001u);
        large |= large_here << (h % 2 * 8);
        if (h % 2 == 1) {
          const int word = (wg * kShare + 16 * h) / 32;
          const uint32_t all = __reduce_and_sync(0xffffffffu, counts ? large : 0xffffffffu);
          if (word < 2 && lane == 0) common[4 * q4 + word] = all;
          large = 0;
        }
      }
      tmem_wait_st();
      tcgen05_fence_before();
      smalls = __reduce_max_sync(0xffffffffu, counts ? smalls : 0u);
      if (lane == 0) common[4 * q4 + 2 + wg] = smalls;
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(q_full);
        mbar_arrive(raw_empty);
      }
      return true;
    };
    int row_exp = 0, row_exp_next = 0;
    bool ok = r0 >= r1 || put_q(0, r0 / p.tiles % p.bands, row_exp_next);
    uint32_t seg = 0, ph_b = 0, ph_add = 0;  // of the score tile that is next, and of the one whose O is
    int b = 0, b_add = 0;
    for (int r = r0; r < r1 && ok; ++seg) {
      const int item = r / p.tiles, head = item / p.bands, band = item - head * p.bands;
      const int t_begin = r - item * p.tiles;
      const int seg_end = min(r1, (item + 1) * p.tiles);
      const int row = band * 128 + row_local;
      row_exp = row_exp_next;
      // this warp group's share of a tile's keys and of the output columns
      constexpr int kKeys = KT / kGroups, kCols = DVP / kGroups, kWords = (kKeys + 31) / 32;
      float2 acc2[kCols / 2];
#pragma unroll
      for (int j = 0; j < kCols / 2; ++j) acc2[j] = make_float2(0.f, 0.f);
      auto add_tile = [&](int g, int e) -> bool {  // O of tile g, whose v has the exponent e
        if (!mbar_wait(pv_done(b_add), ph_add, abort_flag, p.status, 20)) return false;
        if (++b_add == kTiles) { b_add = 0; ph_add ^= 1u; }
        __syncwarp();
        tcgen05_fence_after();
        const float f = power_of_two(row_exp + e);
        uint32_t o[kCols];
#pragma unroll
        for (int h = 0; h < kCols / 8; ++h) tmem_ld8(lanes + kO + (g & 1) * DVP + wg * kCols + h * 8, &o[8 * h]);
        tmem_wait_ld();
#pragma unroll
        for (int j = 0; j < kCols / 2; ++j)
          acc2[j] = ffma2(make_float2(__uint_as_float(o[2 * j]), __uint_as_float(o[2 * j + 1])), make_float2(f, f), acc2[j]);
        tcgen05_fence_before();
        return true;
      };
      const int tiles_here = seg_end - r, g0 = r - r0;
      // the row's mask bits of this share of a tile
      const uint32_t* bits = p.bits + band * 128 + row_local;
      auto mask_of = [&](int t, int i) -> uint32_t {
        const int key = (t_begin + t) * KT + wg * kKeys + 32 * i, word = key >> 5;
        return t < tiles_here && word < p.words ? __ldg(bits + static_cast<size_t>(word) * p.mp) >> (key & 31) : 0u;
      };
      const uint4* tile_info = p.tile_info + head * p.tiles + t_begin;
      uint32_t w[kWords];
#pragma unroll
      for (int i = 0; i < kWords; ++i) w[i] = mask_of(0, i);
      int e_before = 0, e_now = Tile::exponent(__ldcg(&tile_info->x));
      for (int t = 0; t < tiles_here; ++t) {
        const int g = g0 + t;
        uint32_t next[kWords];
#pragma unroll
        for (int i = 0; i < kWords; ++i) next[i] = mask_of(t + 1, i);
        const int e_next = Tile::exponent(__ldcg(&tile_info[min(t + 1, tiles_here - 1)].x));
        if (!mbar_wait(s_full(b), ph_b, abort_flag, p.status, 20)) { ok = false; break; }
        __syncwarp();
        tcgen05_fence_after();
        const uint32_t s_addr = lanes + kS + b * KT + wg * kKeys;
        // 32 keys at a time, over their columns of S: 8 of heads, 8 of tails, twice.  A loop: the warps wait for instructions too
        // (half a warp per issue), and the 64 keys of a tile in one run are 1 to 2 % slower (24 heads x 4096, d 64: 283.4 us a
        // call, 278.5 so).
#pragma unroll 1
        for (int i = 0; i < kWords; ++i) {
          uint32_t x[32];
          tmem_ld32(s_addr + i * 32, x);
          const uint32_t word = i == 0 ? w[0] : w[kWords - 1];
          tmem_wait_ld();
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            uint32_t r[16];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const int c = 16 * h + 2 * j;
              const float a0 = (word & (1u << c)) ? __uint_as_float(x[c]) : 0.f;
              const float a1 = (word & (2u << c)) ? __uint_as_float(x[c + 1]) : 0.f;
              split2(make_float2(a0, a1), r[j], r[8 + j]);
            }
            tmem_st16(s_addr + i * 32 + h * 16, r);
          }
        }
        tmem_wait_st();
        tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(p_full(b));
        if (++b == kTiles) { b = 0; ph_b ^= 1u; }
        // q has been read when the band's last S is there: the next band's goes in under the last PV
        if (t + 1 == tiles_here && seg_end < r1 && !put_q(seg + 1, band + 1 == p.bands ? 0 : band + 1, row_exp_next)) { ok = false; break; }
        if (t > 0 && !add_tile(g - 1, e_before)) { ok = false; break; }
#pragma unroll
        for (int i = 0; i < kWords; ++i) w[i] = next[i];
        e_before = e_now;
        e_now = e_next;
      }
      if (!ok) break;
      if (!add_tile(g0 + tiles_here - 1, e_before)) { ok = false; break; }
      float acc[kCols];
#pragma unroll
      for (int j = 0; j < kCols / 2; ++j) {
        acc[2 * j] = acc2[j].x;
        acc[2 * j + 1] = acc2[j].y;
      }
      bool write = true, look = false;
      if (tiles_here != p.tiles) {
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
        // what warp 3 has found out about this piece is counted with it, in the upper half
        const int which = r == r0 ? 0 : 1;
        if (!mbar_wait(looked_at + 8u * which, 0, abort_flag, p.status, 20)) { ok = false; break; }
        int there = 0;
        if (lane == 0) {
          const int mine = piece[which] >> q4 & 1u ? 0x10001 : 1;
          there = atomicAdd(p.counters + item * 4 * kGroups + wg * 4 + q4, mine) + (mine & 0x10000);
        }
        there = __shfl_sync(0xffffffffu, there, 0);
        write = (there & 0xffff) == last - first;
        look = write && there > 0xffff;
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
        float* dst = p.out + (static_cast<size_t>(head) * p.m + row) * p.dv + wg * kCols;
#pragma unroll
        for (int j = 0; j < kCols / 4; ++j)
          if (wg * kCols + 4 * j < p.dv)
            reinterpret_cast<float4*>(dst)[j] = make_float4(acc[4 * j], acc[4 * j + 1], acc[4 * j + 2], acc[4 * j + 3]);
      }
      if (look) {  // the other warp of the quarter may be another block's; the later one sees to the rows
        __threadfence();
        __syncwarp();
        if (lane == 0 && (atomicXor(p.quarters + item, 16u << q4) >> (4 + q4) & 1u)) atomicOr(again, (r == r0 ? 1u : 16u) << q4);
      }
      r = seg_end;
    }
  }
  tcgen05_fence_before();
  __syncthreads();
  if (warp == 1) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
  const uint32_t cut = *again;
  if (cut != 0 && *abort_flag == 0) {
    static_assert(kAgainWords * 16 <= kRing, "the rings and q are free by now");
    sum_again(p, r0, r1, cut, reinterpret_cast<uint4*>(base_ptr));
  }
}

// 512 threads hold 2 (64 keys) to 4 rows of 16 bytes of k and of v each: with 256 the loads of a block's second half wait behind
// its first (24 heads x 4096, d 64, whole call 283 us, with 512 279, with 1024 284; 6 x 1003, d 80 23.5 and 22.5; 12 x 300 x
// 3000, d 128 47.0, 44.9 and 49.1).
constexpr int kPrepThreads = 512;

// Block (x, h): key tile x of head h as head / tail planes, [2][heads * np][dk] and [2][heads * np][dvk], zeros past n, d and
// dv.  16 threads a row, everything read once and kept in registers.  A row of k is scaled to a largest magnitude in
// [2^kRowExp, 2^(kRowExp + 1)); v takes the factor that k's row lost, and the tile's rows of v together another (exponent).
// Keys where that leaves an element of v too few bits, or that have values of v that are not finite, which are stored as zeros, are
// marked.  And the columns of k are described (Tile).  The blocks of the
// last y zero the main kernel's counters.
template <int kVecs, int KT>
__global__ void __launch_bounds__(kPrepThreads)
attention_prepare_kernel(const AttnParams p, int dk, int dvk, __half* __restrict__ k_planes, __half* __restrict__ v_planes,
                         uint4* __restrict__ tile_info, uint32_t* __restrict__ odd_keys) {
  constexpr int kSide = kPrepThreads / 16, kRows = KT / kSide, kNone = -100000;
  static_assert(kSide == 32, "the keys of a block's i-th rows are a word of odd_keys");
  __shared__ int top_exp, most_small;
  __shared__ uint32_t odd_words[kRows], all_large[2];
  if (threadIdx.x == 0) { top_exp = kNone; most_small = 0; }
  if (threadIdx.x < 2) all_large[threadIdx.x] = 0xffffffffu;
  if (threadIdx.x < kRows) odd_words[threadIdx.x] = 0;
  grid_dependency_wait();
  grid_launch_dependents();
  if (static_cast<int>(blockIdx.y) == p.heads) {
    const int items = p.heads * p.bands;
    for (int i = blockIdx.x * kPrepThreads + threadIdx.x; i < items * 4 * kGroups; i += gridDim.x * kPrepThreads) {
      p.counters[i] = 0;
      if (i < 4 * items) p.odd_rows[i] = 0;
      if (i < items) p.quarters[i] = 0;
    }
    return;
  }
  const int head = blockIdx.y, key0 = blockIdx.x * KT, group = threadIdx.x >> 4, lane16 = threadIdx.x & 15;
  const float* k = p.k + static_cast<size_t>(head) * p.n * p.d;
  const float* v = p.v + static_cast<size_t>(head) * p.n * p.dv;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  float4 xk[kRows][kVecs], xv[kRows][kVecs];
#pragma unroll
  for (int i = 0; i < kRows; ++i) {
    const int key = key0 + group + kSide * i;
#pragma unroll
    for (int j = 0; j < kVecs; ++j) {
      const int c = (lane16 + 16 * j) * 4;
      xk[i][j] = key < p.n && c < p.d ? __ldg(reinterpret_cast<const float4*>(k + static_cast<size_t>(key) * p.d + c)) : zero;
      xv[i][j] = key < p.n && c < p.dv ? __ldg(reinterpret_cast<const float4*>(v + static_cast<size_t>(key) * p.dv + c)) : zero;
    }
  }
  __syncthreads();
  int ek[kRows], top = kNone;
#pragma unroll
  for (int i = 0; i < kRows; ++i) {
    uint32_t bk = 0, bv = 0;
#pragma unroll
    for (int j = 0; j < kVecs; ++j) {
      const float4 a = xk[i][j], b = xv[i][j];
      bk = finite_max(finite_max(finite_max(finite_max(bk, a.x), a.y), a.z), a.w);
      bv = finite_max(finite_max(finite_max(finite_max(bv, b.x), b.y), b.z), b.w);
    }
#pragma unroll
    for (int s = 8; s >= 1; s >>= 1) {
      bk = max(bk, __shfl_xor_sync(0xffffffffu, bk, s));
      bv = max(bv, __shfl_xor_sync(0xffffffffu, bv, s));
    }
    ek[i] = bk != 0u ? exponent_of(bk) : kNone;
    if (bk != 0u && bv != 0u) top = max(top, ek[i] + exponent_of(bv));
  }
  if (lane16 == 0 && top != kNone) atomicMax(&top_exp, top);
  __syncthreads();
  const int exponent = top_exp == kNone ? 0 : top_exp - kTileExp;
  const size_t row0 = static_cast<size_t>(head) * p.np + key0, rows = static_cast<size_t>(p.heads) * p.np;
  auto put = [&](__half* planes, int width, int row, int c, const float4& x, uint2& hi) {
    uint2 lo;
    split2(make_float2(x.x, x.y), hi.x, lo.x);
    split2(make_float2(x.z, x.w), hi.y, lo.y);
    if (c >= width) return;
    __half* dst = planes + (row0 + row) * width + c;
    *reinterpret_cast<uint2*>(dst) = hi;
    *reinterpret_cast<uint2*>(dst + rows * width) = lo;
  };
  uint2 large = make_uint2(0xffffffffu, 0xffffffffu);  // whether this thread's first four columns of k are, in all its rows
  __half2 least = __float2half2_rn(1.f);               // least magnitudes in them
#pragma unroll
  for (int i = 0; i < kRows; ++i) {
    const Scale scale_k(kRowExp - ek[i]), scale_v(ek[i] - exponent);
    const bool none = ek[i] == kNone;  // a row of k that is zero: nothing of v's counts, if it is finite
    bool odd = false;
    auto scaled = [&](float x) -> float {
      const float w = none ? 0.f : scale_v(x);
      const bool finite = isfinite(x);
      odd = odd || !finite || (fabsf(w) < kSmallV && x != 0.f && !none);
      return finite ? w : 0.f;
    };
#pragma unroll
    for (int j = 0; j < kVecs; ++j) {
      const int c = (lane16 + 16 * j) * 4, row_in_tile = group + kSide * i;
      const float4 b = xv[i][j];
      uint2 hi;
      put(k_planes, dk, row_in_tile, c, scaled4(scale_k, xk[i][j]), hi);
      const __half2 x = __habs2(*reinterpret_cast<const __half2*>(&hi.x)), y = __habs2(*reinterpret_cast<const __half2*>(&hi.y));
      if (!none) {
        if (j == 0) {
          large.x &= __hge2_mask(x, __float2half2_rn(kLarge));
          large.y &= __hge2_mask(y, __float2half2_rn(kLarge));
        }
        if (c < p.d) least = __hmin2(least, __hmin2(x, y));
      }
      put(v_planes, dvk, row_in_tile, c, make_float4(scaled(b.x), scaled(b.y), scaled(b.z), scaled(b.w)), hi);
    }
    const uint32_t both = __ballot_sync(0xffffffffu, odd);  // two keys a warp
    if (both != 0 && (threadIdx.x & 31) == 0)
      atomicOr(&odd_words[i], (both & 0xffffu ? 1u << group : 0u) | (both >> 16 ? 2u << group : 0u));
  }
  if (__any_sync(0xffffffffu, __low2float(least) < kSmall || __high2float(least) < kSmall)) {  // rare
    int most = 0;
#pragma unroll
    for (int i = 0; i < kRows; ++i) {
      const Scale scale_k(kRowExp - ek[i]);
      int small = 0;
#pragma unroll
      for (int j = 0; j < kVecs; ++j) {
        const float4 a = scaled4(scale_k, xk[i][j]);
        if ((lane16 + 16 * j) * 4 < p.d && ek[i] != kNone)
          small += (fabsf(a.x) < kSmall ? 1 : 0) + (fabsf(a.y) < kSmall ? 1 : 0) + (fabsf(a.z) < kSmall ? 1 : 0) + (fabsf(a.w) < kSmall ? 1 : 0);
      }
#pragma unroll
      for (int s = 8; s >= 1; s >>= 1) small += __shfl_xor_sync(0xffffffffu, small, s);
      most = max(most, small);
    }
    if (lane16 == 0) atomicMax(&most_small, most);
  }
  uint32_t word = ((large.x & 0x00010001u) | (large.y & 0x00010001u) << 1) << (2 * (lane16 & 7));
#pragma unroll
  for (int s = 4; s >= 1; s >>= 1) word |= __shfl_xor_sync(0xffffffffu, word, s);
  if ((lane16 & 7) == 0) atomicAnd(&all_large[lane16 >> 3], word);
  __syncthreads();
  // A tile that no row of q is safe with: whoever looks at pairs finds its keys' words here, since a block that makes a head's own takes
  // 100 us for it (24 heads x 4096, d 64, q and k after a ReLU: 523 -> 437 us at 5 %, 500 -> 385 at 1 %).
  const int large_columns = __popc(all_large[0]) + __popc(all_large[1]);
  const bool described = 4 * large_columns < min(p.d, 64) || 8 * most_small > large_columns;
  if (described) {
#pragma unroll
    for (int i = 0; i < kRows; ++i) {
      const Scale scale_k(kRowExp - ek[i]);
      const uint4 words = big_and_there(scaled4(scale_k, xk[i][0]), kVecs > 1 ? scaled4(scale_k, xk[i][kVecs - 1]) : zero);
      const int key = key0 + group + kSide * i;
      if (lane16 == 0 && key < p.n) p.key_words[static_cast<size_t>(head) * p.np + key] = words;
    }
  }
  if (threadIdx.x == 0) {
    uint32_t any = 0;
#pragma unroll
    for (int i = 0; i < kRows; ++i) {
      odd_keys[(head * p.np + key0) / 32 + i] = odd_words[i];
      any |= odd_words[i];
    }
    tile_info[head * p.tiles + blockIdx.x] = Tile::pack(exponent, any != 0, most_small, all_large[0], all_large[1], described);
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
  int q, kt, dvp;      // the kernel's template arguments
  int dk, dvk, np, mp;  // row lengths of the planes, keys of a head in them, rows of the mask words
  int tiles;
};

bool attention_shape(int heads, int m, int n, int d, int dv, Shape* s) {
  if (heads < 1 || m < 1 || n < 1 || d < 4 || dv < 4 || d % 4 != 0 || dv % 4 != 0 || d > 128 || dv > 128) return false;
  // A row of all heads' q is a TMA coordinate, a 32-bit integer, and so is the last row of a band that starts inside.
  if (static_cast<long long>(heads) * m > 0x7fffffffll - 128) return false;
  s->q = d <= 64 ? 64 : 128;
  s->dvp = (dv + 31) / 32 * 32;
  s->kt = s->q == 64 && s->dvp <= 64 ? 128 : 64;
  s->dk = (d + 15) / 16 * 16;
  s->dvk = (dv + 15) / 16 * 16;
  s->tiles = (n + s->kt - 1) / s->kt;
  s->np = s->tiles * s->kt;
  s->mp = (m + 127) / 128 * 128;
  const long long tiles = static_cast<long long>(heads) * ((m + 127) / 128) * s->tiles;
  return tiles < (1ll << 30) && 2ll * heads * s->np < (1ll << 30) && heads <= 65000;
}

// One CTA per SM with an equal share of the tiles; with fewer bands than SMs, as many equal pieces of every band as
// fit on the chip, for a CTA that works on two bands pays for a second start (5 us), and no more than this
// root, since whoever comes last adds the pieces up alone.
int cta_count(int items, int tiles, int sms) {
  const int pieces = std::max(1, static_cast<int>(std::sqrt(1.5 * tiles)));
  return items >= sms ? sms : items * std::min(pieces, sms / items);
}

// Times in microseconds, fitted on B200 to 50 measurements: 1 to 32 heads, 256 to 16384 rows and keys, 32 to 128 columns;
// 8 % off (root mean square), 27 % at most.
//
// This kernel multiplies every tile, empty or not: m * n counts, not the positions.  What takes long runs at a lower clock (at
// the power limit) and shares L2: up to 1.7 times as long for the same tiles.
double one_launch_us(int heads, int m, int n, const Shape& s, int sms) {
  const int bands = (m + 127) / 128, items = heads * bands;
  const int ctas = cta_count(items, s.tiles, sms);
  const double tile = 0.57 + 2.5e-5 * (s.dk + s.dvk) * s.kt;
  const double planes = 1.8e-6 * heads * n * (s.dk + s.dvk);
  const double cool = planes + (static_cast<long long>(items) * s.tiles + ctas - 1) / ctas * tile;
  return 18.0 + cool * (1.0 + 0.7 * cool / (cool + 240.0));
}

// SDDMM and SpMM head by head over two streams (pytorch/attention.py), fitted to 578 measurements with masks of 0.05 to
// 23 % stored positions, scattered or in a band: 20 us of host time a head for the two launches, or
// what their gathers take, which follows the positions (a row of q.k and of v for each), and the dense tiles of the SDDMM
// where that is the tensor-core one.
double head_by_head_us(int heads, int m, int n, int d, int dv, int nnz) {
  auto row = [](int cols) { return cols <= 32 ? 32 : cols <= 64 ? 64 : 128; };
  double head = (0.6e-5 + 0.235e-6 * (row(d) + row(dv))) * nnz;
  if (iex_sddmm_f32_prefers_tc(m, d, n, nnz, 1)) head += 0.4e-6 * m * n;
  return std::max(28.0 + 19.5 * heads, 10.0 + heads * head);
}

size_t round256(size_t v) { return (v + 255) & ~static_cast<size_t>(255); }

template <int kQ, int KT, int DVP>
int launch_attention(const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, const AttnParams& p, int ctas,
                     cudaStream_t s) {
  auto kern = attention_kernel<kQ, KT, DVP>;
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
  return launch_overlapped(kern, dim3(ctas), dim3(kThreads), static_cast<size_t>(227 * 1024), s, mq, mk, mv, p);
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

// One launch where it is estimated faster than the operators: of the 50 measurements 49 are, a tie goes the other way.  Measured (us,
// one launch / head by head): 4096 x 4096, 12 heads, d 64: 139 / 269 at 2 %; d 80: 213 / 258 at 0.2 %, 222 / 698 at 5 %; 32 heads,
// d 128: 785 / 780 at 2 %, 772 / 3514 at 10 %; 16384 x 16384, 1 head, d 64: 162 / 50 for a band of 32; 32 heads x 8192, d 64:
// 1517 / 635 at 0.2 %; 6314 x 6314, 1 head, d 32: 41 / 50 at 1 %.
extern "C" int iex_attention_f32_prefers(int heads, int m, int n, int d, int dv, int nnz) {
  Shape s;
  if (!attention_shape(heads, m, n, d, dv, &s)) return 0;
  return one_launch_us(heads, m, n, s, std::min(sm_count(), kNumSMs)) <= head_by_head_us(heads, m, n, d, dv, nnz);
}

// Whether a mask of this size and number of stored positions has up to 64 heads of some widths that prefer one launch.  The widths
// are the least of every class that the operators' time has, where the launch is cheapest; a tensor-core SDDMM takes 32 and 64
// alone.  25 us on the host where nothing does.
extern "C" int iex_attention_f32_may_prefer(int m, int n, int nnz) {
  for (int d : {4, 36, 68, 32, 64})
    for (int dv : {4, 36, 68})
      for (int heads = 1; heads <= 64; ++heads)
        if (iex_attention_f32_prefers(heads, m, n, d, dv, nnz)) return 1;
  return 0;
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

namespace {

// Sections of the workspace, each on 256 bytes.
struct Sections {
  size_t k, v, tile_info, odd_keys, key_words, partials, counters, quarters, odd_rows, end;
  Sections(int heads, int m, const Shape& s) {
    const size_t rows = 2ull * heads * s.np, tiles = 16ull * heads * s.tiles, items = static_cast<size_t>(heads) * ((m + 127) / 128);
    k = 0;
    v = k + round256(rows * s.dk * 2);
    tile_info = v + round256(rows * s.dvk * 2);
    odd_keys = tile_info + round256(tiles);
    key_words = odd_keys + round256(rows / 16);
    partials = key_words + round256(rows * 8);
    counters = partials + round256(2ull * kNumSMs * 128 * s.dvp * 4);
    quarters = counters + round256(16 * kGroups * items);
    odd_rows = quarters + round256(4 * items);
    end = odd_rows + round256(16 * items);
  }
};

}  // namespace

extern "C" size_t iex_attention_workspace_bytes(int heads, int m, int n, int d, int dv) {
  Shape s;
  if (!attention_shape(heads, m, n, d, dv, &s)) return 0;
  return Sections(heads, m, s).end;
}

extern "C" int iex_attention_f32(int heads, int m, int n, int d, int dv, const void* plan, const int32_t* row_offsets,
                                 const int32_t* column_indices, const float* q, const float* k, const float* v, float* out,
                                 void* workspace, size_t workspace_bytes, void* stream) {
  if (heads < 0 || m < 0 || n < 0 || d < 0 || dv < 0) return IEX_ERR_BAD_ARG;
  if (heads == 0 || m == 0 || dv == 0) return IEX_OK;
  Shape s;
  if (!attention_shape(heads, m, n, d, dv, &s)) return IEX_ERR_UNSUPPORTED;
  if (!plan || !row_offsets || !column_indices || !q || !k || !v || !out || !workspace) return IEX_ERR_BAD_ARG;
  const Sections at(heads, m, s);
  if (workspace_bytes < at.end) return IEX_ERR_TOO_LARGE;
  if (!aligned16(q) || !aligned16(k) || !aligned16(v) || !aligned16(out) || (reinterpret_cast<uintptr_t>(workspace) & 255u))
    return IEX_ERR_UNSUPPORTED;
  uint8_t* ws = static_cast<uint8_t*>(workspace);
  __half* k_planes = reinterpret_cast<__half*>(ws + at.k);
  __half* v_planes = reinterpret_cast<__half*>(ws + at.v);
  uint4* tile_info = reinterpret_cast<uint4*>(ws + at.tile_info);
  uint32_t* odd_keys = reinterpret_cast<uint32_t*>(ws + at.odd_keys);
  AttnParams p{};
  p.partials = reinterpret_cast<float4*>(ws + at.partials);
  p.counters = reinterpret_cast<int*>(ws + at.counters);
  p.odd_rows = reinterpret_cast<uint32_t*>(ws + at.odd_rows);
  p.quarters = reinterpret_cast<uint32_t*>(ws + at.quarters);
  p.heads = heads; p.m = m; p.n = n; p.d = d; p.dv = dv;
  p.bands = (m + 127) / 128;
  p.tiles = s.tiles;
  p.mp = s.mp;
  p.np = s.np;
  p.words = (n + 31) / 32;
  p.total = heads * p.bands * p.tiles;
  p.bits = static_cast<const uint32_t*>(plan) + 64;
  p.q = q; p.k = k; p.v = v; p.out = out;
  p.row_offsets = row_offsets;
  p.cols = column_indices;
  p.tile_info = tile_info;
  p.odd_keys = odd_keys;
  p.key_words = reinterpret_cast<uint4*>(ws + at.key_words);
  p.status = status_word();
  const int sms = std::min(sm_count(), kNumSMs), ctas = cta_count(heads * p.bands, p.tiles, sms);
  CUtensorMap mq, mk, mv;
  int st = make_map_f32(&mq, q, static_cast<long long>(heads) * m, d, 128);
  if (st == IEX_OK) st = make_map_f16(&mk, k_planes, 2ll * heads * s.np, s.dk, s.dk, s.kt, 64, true);
  if (st == IEX_OK) st = make_map_f16(&mv, v_planes, 2ll * heads * s.np, s.dvk, s.dvk, s.kt, 64, true);
  if (st != IEX_OK) return st;
  cudaStream_t cs = static_cast<cudaStream_t>(stream);
  // The prepare kernel of a call usually follows the main kernel of the one before.  Launched ahead of that kernel's end its
  // blocks would crowd on the few SMs that are free (6 heads x 1003, d 80: 42 us a call instead of 31), so that is
  // done only where main kernels leave a third of the chip free (then it saves 1 to 2 us).
  const dim3 prep_grid(p.tiles, heads + 1);
  auto prepare = s.kt == 128 ? attention_prepare_kernel<1, 128> : attention_prepare_kernel<2, 64>;
  if (3 * ctas <= 2 * sms) {
    st = launch_overlapped(prepare, prep_grid, dim3(kPrepThreads), 0, cs, p, s.dk, s.dvk, k_planes, v_planes, tile_info, odd_keys);
  } else {
    prepare<<<prep_grid, kPrepThreads, 0, cs>>>(p, s.dk, s.dvk, k_planes, v_planes, tile_info, odd_keys);
    st = launch_status();
  }
  if (st != 0) return st;
  const int which = s.q + s.dvp / 32;
  switch (which) {
    case 65: return launch_attention<64, 128, 32>(mq, mk, mv, p, ctas, cs);
    case 66: return launch_attention<64, 128, 64>(mq, mk, mv, p, ctas, cs);
    case 67: return launch_attention<64, 64, 96>(mq, mk, mv, p, ctas, cs);
    case 68: return launch_attention<64, 64, 128>(mq, mk, mv, p, ctas, cs);
    case 129: return launch_attention<128, 64, 32>(mq, mk, mv, p, ctas, cs);
    case 130: return launch_attention<128, 64, 64>(mq, mk, mv, p, ctas, cs);
    case 131: return launch_attention<128, 64, 96>(mq, mk, mv, p, ctas, cs);
    case 132: return launch_attention<128, 64, 128>(mq, mk, mv, p, ctas, cs);
    default: return IEX_ERR_UNSUPPORTED;
  }
}
