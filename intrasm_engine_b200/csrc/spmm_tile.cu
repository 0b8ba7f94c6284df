// fp16 CSR SpMM on tensor cores by decoding the matrix tile by tile into shared memory, alone or
// in one launch with a dense linear on the same activations (the fused sparse || dense layer):
//   sparse   S[r, t] = sum_p values[p] * X[col[p], t]         dense   D[f, t] = sum_c W[f, c] * X[c, t]
//
// A unit of work is a run of rows of either matrix over the whole K range, one unit per CTA
// where there are enough SMs.  For tcgen05.mma the activations are the M operand (64 or 128 tokens) and the
// unit's rows the N operand, so a unit may have any multiple of 8 rows: the rows are
// dealt out so that every SM gets one unit and all finish together (plan_tile).
//
//   warp 0       TMA producer: 64-column slots of X (either storage order), and of W for dense units
//   warp 1       MMA issuer
//   warps 2-21   sparse units: CSR decoders.  Each owns rows of the unit.  Block by block (kb columns,
//                two buffers) a warp clears its rows of the buffer and scatters their nonzeros into
//                the 128-byte-swizzled K-major layout; MMA of one block runs under the decoding of
//                the next.  After the last block they read the accumulator out.
//
// What bounds a sparse unit is instruction issue in the decoders, so the inner loop is built for few
// instructions per nonzero: neighbouring lanes take neighbouring pairs of nonzeros straight from
// global memory (4-byte loads, U pairs per lane requested one row ahead, and an L2 prefetch further
// ahead), both columns of a pair are turned into shared-memory offsets by the same packed 16-bit
// operations, and because columns ascend the two-byte stores of a warp spread over the banks.  A
// row's position after a block is a count of the columns below the block's end (ballots): no
// search, no per-tile metadata, and no synchronisation between warps except one arrival per block.
// The tile decoder it replaces kept eight 64-column slots open and re-read and re-checked every
// row in rounds of dependent steps: 11008 x 4096 x 64 tokens 45.7 -> 42.3 us at 50 %, 29.6 -> 22.6 us at 90 %.  16 or 24
// decoders are slower than 20 (registers; issue slots).
//
// Row groups of 8 hold their 64-column atoms next to each other (descriptor stride kb / 64 KB), so
// that a column's offset inside a row group is two bit fields of the column and no multiplication.
//
// Every mbarrier wait is bounded, as in tc_fused.cu.
#include <cuda.h>

#include <cmath>
#include <mutex>

#include "common.cuh"
#include "csr_terms.cuh"
#include "tc_ptx.cuh"

namespace iex {
namespace tc {

int make_map_f16(CUtensorMap* map, const void* base, long long rows, long long cols, long long ld, int box_rows,
                 int box_cols, bool swizzle);  // tc_fused.cu

namespace {

constexpr int kDecoders = 20;    // 24 warps' worth of registers: 80 a thread; 16 and 24 decoders measured slower
constexpr int kThreads = (2 + kDecoders) * 32;
constexpr int kMaxXSlots = 4;    // sparse units: slots of X
constexpr int kMaxStages = 8;    // dense units: slots of X and W together
constexpr int kBars = 2 * kMaxXSlots + 4 + 2 * kMaxStages + 1;
constexpr int kBarBytes = 8 * kBars + 16;
constexpr int kBudget = (227 * 1024 - 1024 - kBarBytes) & ~1023;

struct TileParams {
  // sparse units: s_tiles runs of s_rows rows; out[r * s_row + t * s_tok]
  int s_tiles, s_rows, s_m, s_nnz;
  const int* row_offsets;
  const void* cols;
  const __half* values;
  const float* bias;  // optional: relu(sum + bias[row])
  __half* s_out;
  long long s_row, s_tok;
  // dense units of one or two matrices on the same activations, d_rows rows each
  int d_rows;
  int d_tiles[2], d_m[2];
  __half* d_out[2];
  long long d_row[2], d_tok[2];
  // shared
  int k, n;
  int x_mn;            // X stored [k, n] (tokens contiguous), else [n, k]
  int inst_m;          // tokens per MMA: 64 or 128
  int m_blocks;        // 1 or 2 of them
  int kb;              // columns per sparse block, a multiple of 64 up to 512
  int x_slots, stages;
  int acc_cols, tmem_cols;
  int ahead;           // nonzeros of L2 prefetch distance
  CsrTerms terms;      // of the sparse units, or of the first dense matrix where that is a CSR matrix's dense copy
  int* status;
};

__device__ __forceinline__ void umma(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(acc)
      : "memory");
}

// This thread's outputs of a unit whose matrix is a CSR one, for token t_local and, if the bits say so, the one inst_m further: summed again
// (csr_terms.cuh) and stored over what is there.  Called with next to nothing live: the decoders have no registers to spare.
__device__ __noinline__ void store_again(const TileParams& p, int row0, int rows, int first, int t_local, uint32_t blocks) {
  for (int mb = 0; mb < p.m_blocks; ++mb) {
    const int t = mb * p.inst_m + t_local;
    if (!(blocks >> mb & 1u) || t >= p.n) continue;
    for (int c = first; c < rows; c += kDecoders * 8)
      for (int row = row0 + c; row < min(row0 + min(c + 32, rows), p.s_m); ++row) {
        float v = sum_stored(p.terms, row, t);
        if (p.bias != nullptr) v = fmaxf(v + __ldg(p.bias + row), 0.f);
        p.s_out[row * p.s_row + t * p.s_tok] = __float2half_rn(v);
      }
  }
}

// U pairs of a lane as loaded, the columns in the matrix's index type.  A half warp (16 lanes) reads one
// row: pair u of its lane h are positions base + 32 u + 2 h and the next.
template <typename IT, int U> struct Window;
template <int U> struct Window<uint16_t, U> { uint32_t v[U], c[U]; };
template <int U> struct Window<int, U> { uint32_t v[U]; int2 c[U]; };

// Requests positions [base, base + 32 U) of the arrays, whatever row they belong to.
template <typename IT, int U>
__device__ __forceinline__ void load_window(Window<IT, U>& w, const __half* __restrict__ values,
                                            const IT* __restrict__ cols, int base, int half_lane) {
  const __half* pv = values + base + 2 * half_lane;
  const IT* pc = cols + base + 2 * half_lane;
#pragma unroll
  for (int u = 0; u < U; ++u) {
    w.v[u] = __ldg(reinterpret_cast<const uint32_t*>(pv + 32 * u));
    if constexpr (sizeof(IT) == 2) w.c[u] = __ldg(reinterpret_cast<const uint32_t*>(pc + 32 * u));
    else w.c[u] = __ldg(reinterpret_cast<const int2*>(pc + 32 * u));
  }
}
// Gives the positions of a window outside [cur, end) an index no block contains.
template <int U>
__device__ __forceinline__ void cut_window(Window<uint16_t, U>& w, int p0, int cur, int end) {
  const uint32_t n = static_cast<uint32_t>(end - cur), q = static_cast<uint32_t>(p0 - cur);
#pragma unroll
  for (int u = 0; u < U; ++u) {
    w.c[u] |= q + 32u * u >= n ? 0x0000ffffu : 0u;
    w.c[u] |= q + 32u * u + 1u >= n ? 0xffff0000u : 0u;
  }
}
template <int U>
__device__ __forceinline__ void cut_window(Window<int, U>& w, int p0, int cur, int end) {
  const uint32_t n = static_cast<uint32_t>(end - cur), q = static_cast<uint32_t>(p0 - cur);
#pragma unroll
  for (int u = 0; u < U; ++u) {
    w.c[u].x = q + 32u * u >= n ? -1 : w.c[u].x;
    w.c[u].y = q + 32u * u + 1u >= n ? -1 : w.c[u].y;
  }
}
// Both columns of pair u relative to the block's first column, 16 bits each.  Columns ascend and everything
// before the row's position is masked (`before`), so no column is below the block's first one.
template <int U>
__device__ __forceinline__ uint32_t relative(const Window<uint16_t, U>& w, int u, uint32_t c0c0, uint32_t before) {
  return (u == 0 ? w.c[0] | before : w.c[u]) - c0c0;
}
template <int U>
__device__ __forceinline__ uint32_t relative(const Window<int, U>& w, int u, uint32_t c0c0, uint32_t before) {
  const uint32_t c0 = c0c0 & 0xffffu;
  const uint32_t a = min(static_cast<uint32_t>(w.c[u].x) - c0, 0xffffu);
  const uint32_t b = min(static_cast<uint32_t>(w.c[u].y) - c0, 0xffffu);
  return (u == 0 ? a | before : a) | (b << 16);
}
// If key < limit: stores the low half of v at addr and counts it.  Predicated instructions, one
// comparison for both.
__device__ __forceinline__ void store_below(uint32_t key, uint32_t limit, uint32_t addr, uint32_t v, uint32_t& count) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b16 h;\n\t"
      "setp.lt.u32 p, %1, %2;\n\t"
      "cvt.u16.u32 h, %4;\n\t"
      "@p st.shared.u16 [%3], h;\n\t"
      "@p add.u32 %0, %0, 1;\n\t}"
      : "+r"(count)
      : "r"(key), "r"(limit), "r"(addr), "r"(v)
      : "memory");
}

// Offsets of the mbarriers behind `bar`.
constexpr uint32_t kXFull = 0, kXEmpty = 8u * kMaxXSlots, kAFull = 16u * kMaxXSlots, kAEmpty = kAFull + 16u,
                   kDFull = kAFull + 32u, kDEmpty = kDFull + 8u * kMaxStages, kAccFull = kDEmpty + 8u * kMaxStages;

// Everything the MMA thread does for one unit.  It is a serial bottleneck (one thread feeds the
// tensor pipe), so the token blocks and the storage order of X are template parameters: four (eight)
// instructions per slot unrolled over constants.
template <int kMB, bool kXMn>
__device__ __forceinline__ void issue_unit(const TileParams& p, bool sparse, int rows, uint32_t base, uint32_t x_base,
                                           uint32_t x_bytes, uint32_t stage_bytes, uint32_t block_bytes, uint32_t bar,
                                           uint32_t tmem, uint32_t x_it, uint32_t a_it, uint32_t d_it,
                                           volatile int* abort_flag) {
  const uint32_t idesc = (1u << 4) | (kXMn ? (1u << 15) : 0u) | (static_cast<uint32_t>(rows >> 3) << 17) |
                         (static_cast<uint32_t>(p.inst_m >> 4) << 24);
  constexpr uint32_t a_step = kXMn ? 2048u : 32u;   // 16 columns of X further
  constexpr uint32_t mb_step = 128u * 128u;         // the second block of 128 tokens
  const uint32_t tmem1 = tmem + p.acc_cols;
  const int k_slots = (p.k + 63) / 64;
  auto issue = [&](uint32_t x_addr, uint64_t bd, uint32_t acc) {
    const uint64_t ad = kXMn ? smem_desc(x_addr, 8192, 1024) : smem_desc(x_addr, 16, 1024);
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
      umma(tmem, desc_advance(ad, ks * a_step), desc_advance(bd, ks * 32u), idesc, ks == 0 ? acc : 1u);
      if constexpr (kMB == 2) umma(tmem1, desc_advance(ad, mb_step + ks * a_step), desc_advance(bd, ks * 32u), idesc, ks == 0 ? acc : 1u);
    }
  };
  uint32_t acc = 0;
  if (sparse) {
    const int atoms = p.kb / 64, blocks = (p.k + p.kb - 1) / p.kb;
    uint32_t s = x_it % p.x_slots, ph = (x_it / p.x_slots) & 1u;
    for (int b = 0; b < blocks; ++b) {
      const uint32_t ab = a_it + b;
      if (!mbar_wait(bar + kAFull + 8u * (ab & 1u), (ab >> 1) & 1u, abort_flag, p.status, 32)) return;
      uint64_t bd = smem_desc(base + (ab & 1u) * block_bytes, 16, static_cast<uint32_t>(atoms) * 1024u);
      const int slots = min(atoms, k_slots - b * atoms);
      for (int j = 0; j < slots; ++j) {
        if (!mbar_wait(bar + kXFull + 8u * s, ph, abort_flag, p.status, 32)) return;
        tcgen05_fence_after();
        issue(x_base + s * x_bytes, bd, acc);
        umma_commit(bar + kXEmpty + 8u * s);
        acc = 1;
        bd = desc_advance(bd, 1024u);
        if (++s == static_cast<uint32_t>(p.x_slots)) { s = 0; ph ^= 1u; }
      }
      umma_commit(bar + kAEmpty + 8u * (ab & 1u));
    }
  } else {
    uint32_t s = d_it % p.stages, ph = (d_it / p.stages) & 1u;
    for (int ks = 0; ks < k_slots; ++ks) {
      if (!mbar_wait(bar + kDFull + 8u * s, ph, abort_flag, p.status, 32)) return;
      tcgen05_fence_after();
      const uint32_t src = base + s * stage_bytes;
      issue(src, smem_desc(src + x_bytes, 16, 1024), acc);
      umma_commit(bar + kDEmpty + 8u * s);
      acc = 1;
      if (++s == static_cast<uint32_t>(p.stages)) { s = 0; ph ^= 1u; }
    }
  }
  umma_commit(bar + kAccFull);
}

// kSparse false: a launch of dense units only
template <typename IT, int U, bool kSparse = true>
__global__ void __launch_bounds__(kThreads, 1)
spmm_tile_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w0,
                 const __grid_constant__ CUtensorMap map_w1, const __grid_constant__ TileParams p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* base_ptr = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t x_bytes = static_cast<uint32_t>(p.inst_m * p.m_blocks) * 128u;  // one slot of X
  const uint32_t atoms = static_cast<uint32_t>(p.kb) / 64u;
  const uint32_t block_bytes = static_cast<uint32_t>(p.s_rows / 8) * atoms * 1024u;
  const uint32_t x_base = base + 2u * block_bytes;
  const uint32_t w_bytes = static_cast<uint32_t>(p.d_rows) * 128u;
  const uint32_t stage_bytes = x_bytes + w_bytes;
  const uint32_t bar = base + kBudget;
  auto x_full = [&](int s) { return bar + kXFull + 8u * s; };
  auto x_empty = [&](int s) { return bar + kXEmpty + 8u * s; };
  auto a_full = [&](int s) { return bar + kAFull + 8u * s; };
  auto a_empty = [&](int s) { return bar + kAEmpty + 8u * s; };
  auto d_full = [&](int s) { return bar + kDFull + 8u * s; };
  auto d_empty = [&](int s) { return bar + kDEmpty + 8u * s; };
  const uint32_t acc_full = bar + kAccFull;
  volatile uint32_t* tmem_ptr = reinterpret_cast<volatile uint32_t*>(base_ptr + kBudget + 8 * kBars);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_ptr + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kMaxXSlots; ++s) { mbar_init(x_full(s), 1); mbar_init(x_empty(s), 1); }
    for (int s = 0; s < 2; ++s) { mbar_init(a_full(s), kDecoders); mbar_init(a_empty(s), 1); }
    for (int s = 0; s < kMaxStages; ++s) { mbar_init(d_full(s), 1); mbar_init(d_empty(s), 1); }
    mbar_init(acc_full, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(bar + 8u * kBars),
                 "r"(static_cast<uint32_t>(p.tmem_cols))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem = *tmem_ptr;
  grid_dependency_wait();
  grid_launch_dependents();

  const int k_slots = (p.k + 63) / 64;
  const int blocks = (p.k + p.kb - 1) / p.kb;
  const int units = p.s_tiles + p.d_tiles[0] + p.d_tiles[1];
  uint32_t x_it = 0, d_it = 0, a_it = 0;  // slots / stages / blocks used so far (each role counts alike)
  uint32_t unit_it = 0;

  for (int u = blockIdx.x; u < units; u += gridDim.x, ++unit_it) {
    const bool sparse = kSparse && u < p.s_tiles;
    const int rows = sparse ? p.s_rows : p.d_rows;
    const int which = u >= p.s_tiles + p.d_tiles[0] ? 1 : 0;  // dense matrix
    const int row0 = (sparse ? u : u - p.s_tiles - (which ? p.d_tiles[0] : 0)) * rows;
    if (warp == 0) {
      // ---------------------------------------------------------------- TMA producer
      if (elect_one()) {
        const int m_atoms = p.inst_m * p.m_blocks / 64;
        auto load_x = [&](uint32_t dst, uint32_t full, int ks) {
          if (p.x_mn) {
            for (int j = 0; j < m_atoms; ++j) tma_load_2d(dst + j * 8192u, &map_x, full, j * 64, ks * 64);
          } else {
            tma_load_2d(dst, &map_x, full, ks * 64, 0);
          }
        };
        if (sparse) {
          int s = x_it % p.x_slots;
          uint32_t ph = (x_it / p.x_slots) & 1u;
          for (int ks = 0; ks < k_slots; ++ks) {
            if (!mbar_wait(x_empty(s), ph ^ 1u, abort_flag, p.status, 64)) break;
            mbar_arrive_expect_tx(x_full(s), x_bytes);
            load_x(x_base + s * x_bytes, x_full(s), ks);
            if (++s == p.x_slots) { s = 0; ph ^= 1u; }
          }
        } else {
          int s = d_it % p.stages;
          uint32_t ph = (d_it / p.stages) & 1u;
          for (int ks = 0; ks < k_slots; ++ks) {
            if (!mbar_wait(d_empty(s), ph ^ 1u, abort_flag, p.status, 64)) break;
            const uint32_t dst = base + s * stage_bytes;
            mbar_arrive_expect_tx(d_full(s), stage_bytes);
            tma_load_2d(dst + x_bytes, which ? &map_w1 : &map_w0, d_full(s), ks * 64, row0);
            load_x(dst, d_full(s), ks);
            if (++s == p.stages) { s = 0; ph ^= 1u; }
          }
        }
        if (*abort_flag)  // drain: bounded time for the copies this thread armed to land
          for (uint32_t i = 0; i < 2048u; ++i) __nanosleep(100);
      }
      __syncwarp();
    } else if (warp == 1) {
      // ---------------------------------------------------------------- MMA issuer
      if (elect_one()) {
        if (p.m_blocks == 1) {
          if (p.x_mn) issue_unit<1, true>(p, sparse, rows, base, x_base, x_bytes, stage_bytes, block_bytes, bar, tmem, x_it, a_it, d_it, abort_flag);
          else issue_unit<1, false>(p, sparse, rows, base, x_base, x_bytes, stage_bytes, block_bytes, bar, tmem, x_it, a_it, d_it, abort_flag);
        } else {
          if (p.x_mn) issue_unit<2, true>(p, sparse, rows, base, x_base, x_bytes, stage_bytes, block_bytes, bar, tmem, x_it, a_it, d_it, abort_flag);
          else issue_unit<2, false>(p, sparse, rows, base, x_base, x_bytes, stage_bytes, block_bytes, bar, tmem, x_it, a_it, d_it, abort_flag);
        }
      }
      __syncwarp();
    } else {
      // ---------------------------------------------------------------- decoders
      const int w = warp - 2;
      bool ok = true;
      if (sparse) {
        const IT* cols = static_cast<const IT*>(p.cols);
        // The warp's row pairs are w, w + kDecoders, ...: pair d is rows 2 d (lanes 0-15) and 2 d + 1.
        const int pairs = (rows / 2 - w + kDecoders - 1) / kDecoders;
        const int hl = lane & 15, hi = lane >> 4;
        // lane 16 h + i holds the position and the end of row h of the warp's pair i
        int cur_l = 0, end_l = 0;
        if (hl < pairs) {
          const int r = row0 + 2 * (w + kDecoders * hl) + hi;
          if (r < p.s_m) {
            cur_l = __ldg(p.row_offsets + r);
            end_l = __ldg(p.row_offsets + r + 1);
          }
        }
        // Windows are whole pairs inside the arrays: the last ones start early (last_base), and of an odd
        // number of nonzeros the very last is taken out of its row and written by itself.
        const int last_base = (p.s_nnz & ~1) - 32 * U;
        int tail_pair = -1, tail_lane = -1, tail_col = 0;
        uint32_t tail_val = 0;
        if (p.s_nnz & 1) {
          const uint32_t has = __ballot_sync(0xffffffffu, end_l == p.s_nnz && cur_l < end_l);
          if (has != 0) {
            tail_lane = (__ffs(has) - 1) & 16;
            tail_pair = (__ffs(has) - 1) & 15;
            tail_col = to_index(__ldg(cols + p.s_nnz - 1));
            tail_val = __half_as_ushort(__ldg(p.values + p.s_nnz - 1));
            if (hl == tail_pair && hi == tail_lane >> 4) --end_l;
          }
        }
        // L2 prefetch: per half warp up to eight 128-byte lines of values and as many of (16-bit) indices
        const int pf_pos = (lane & 7) * (hl < 8 ? 64 : 128 / static_cast<int>(sizeof(IT)));
        const char* const pf_base = hl < 8 ? reinterpret_cast<const char*>(p.values) : reinterpret_cast<const char*>(cols);
        const int pf_size = hl < 8 ? 2 : static_cast<int>(sizeof(IT));
        const bool pf_on = pf_pos < p.ahead;
        auto prefetch = [&](int from, int end) {
          const int q = from + pf_pos;
          if (pf_on && q < end) asm volatile("prefetch.global.L2 [%0];" ::"l"(pf_base + static_cast<long long>(q) * pf_size));
        };
        const uint32_t kb_hi = static_cast<uint32_t>(p.kb) << 16;
        for (int j = 0; j < pairs; ++j)
          prefetch(__shfl_sync(0xffffffffu, cur_l, (lane & 16) + j), __shfl_sync(0xffffffffu, end_l, (lane & 16) + j));
        // Items: the share of block b in the rows of pair i, row pairs inside blocks.  `win` holds the item's
        // window, `next` the following item's (loaded one item ahead; with a single row pair per warp
        // its position is not known earlier).  The loop is written to have one copy of every part: its
        // instructions have to fit the instruction caches that 20 warps at different places share
        // (two inlined copies of the item: 44 instead of 40 us at 11008 x 4096, 50 %).
        int b = 0, i = 0, li = 0;
        uint32_t buf = 0;
        bool loaded = false;
        Window<IT, U> win, next;
        while (pairs > 0 && b < blocks) {
          if (pairs > 1 || !loaded) {
            const int c = __shfl_sync(0xffffffffu, cur_l, (lane & 16) + li);
            load_window<IT, U>(next, p.values, cols, min(c & ~1, last_base), hl);
            li = li + 1 < pairs ? li + 1 : 0;
          }
          if (!loaded) {
            win = next;
            loaded = true;
            continue;
          }
          const uint32_t ab = a_it + b;
          if (i == 0) {
            buf = base + (ab & 1u) * block_bytes;
            if (!mbar_wait(a_empty(ab & 1u), ((ab >> 1) & 1u) ^ 1u, abort_flag, p.status, 32)) { ok = false; break; }
          }
          int cur = __shfl_sync(0xffffffffu, cur_l, (lane & 16) + i);
          int end = __shfl_sync(0xffffffffu, end_l, (lane & 16) + i);
          const uint32_t r = 2u * (w + kDecoders * i);
          const uint32_t pair_base = buf + (r >> 3) * atoms * 1024u + (r & 7u) * 128u;
          // clear the pair's 256 bytes of every atom: a half warp each, two atoms at a time
          {
            const uint32_t dst = pair_base + hi * 1024u + hl * 16u;
#pragma unroll
            for (uint32_t t = 0; t < 8; t += 2)
              if (t + hi < atoms)
                asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(dst + t * 1024u), "r"(0u) : "memory");
          }
          prefetch(cur + p.ahead, end);
          const uint32_t row_base = pair_base + hi * 128u;
          const uint32_t sw2 = (((r & 7u) + hi) << 4) * 0x00010001u;
          const uint32_t c0 = static_cast<uint32_t>(b * p.kb), c0c0 = c0 * 0x00010001u;
          __syncwarp();
          if (i == tail_pair && lane == tail_lane && static_cast<uint32_t>(tail_col) - c0 < static_cast<uint32_t>(p.kb)) {
            uint32_t one = 0;
            const uint32_t rel = static_cast<uint32_t>(tail_col) - c0;
            store_below(0u, 1u, row_base + (((rel << 4) & 0x1c00u) | (((rel << 1) & 0x7eu) ^ (sw2 & 0xffffu))), tail_val, one);
          }
          for (;;) {
            const int wbase = min(cur & ~1, last_base);
            if (__any_sync(0xffffffffu, wbase + 32 * U > end || wbase + 1 < cur)) cut_window<U>(win, wbase + 2 * hl, cur, end);
            const uint32_t before = (hl == 0 && (cur & 1)) ? 0xffffu : 0u;
            uint32_t cnt = 0;
#pragma unroll
            for (int q = 0; q < U; ++q) {
              const uint32_t rel = relative<U>(win, q, c0c0, before);
              // offset inside the row group: 64-column atom (bits 6-8 of the column) and swizzled byte
              const uint32_t off = ((rel << 4) & 0x1c001c00u) | (((rel << 1) & 0x007e007eu) ^ sw2);
              store_below(rel << 16, kb_hi, row_base + (off & 0xffffu), win.v[q], cnt);
              store_below(rel, kb_hi, row_base + (off >> 16), win.v[q] >> 16, cnt);
            }
            // both rows' counts in one reduction: the upper half warp's in the upper 16 bits
            const uint32_t both = __reduce_add_sync(0xffffffffu, hi ? cnt << 16 : cnt);
            cur += hi ? both >> 16 : both & 0xffffu;
            const bool again = cur == wbase + 32 * U && cur < end;  // the whole window fell into the block
            if (!__any_sync(0xffffffffu, again)) break;
            load_window<IT, U>(win, p.values, cols, min(cur & ~1, last_base), hl);
            if (!again) end = cur;  // this row is done with the block: nothing of the window counts
          }
          if (hl == i) cur_l = cur;
          i = i + 1 < pairs ? i + 1 : 0;
          if (i == 0) {  // the block's last pair of this warp
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(a_full(ab & 1u));
            ++b;
          }
          if (pairs > 1) win = next; else loaded = false;
        }
        if (pairs <= 0) {  // no row of the unit for this warp: only its arrivals
          for (; b < blocks; ++b) {
            const uint32_t ab = a_it + b;
            if (!mbar_wait(a_empty(ab & 1u), ((ab >> 1) & 1u) ^ 1u, abort_flag, p.status, 32)) { ok = false; break; }
            if (lane == 0) mbar_arrive(a_full(ab & 1u));
          }
        }
      }
      // ---------------------------------------------------------------- read-out
      if (ok && mbar_wait(acc_full, unit_it & 1u, abort_flag, p.status, 64)) {
        tcgen05_fence_after();
        const int q = warp & 3, share = w >> 2;  // tensor-memory quarter; the warps of a quarter split its columns
        const int t_local = p.inst_m == 64 ? q * 16 + lane : q * 32 + lane;
        const bool lane_ok = p.inst_m == 128 || lane < 16;
        const int m_rows = sparse ? p.s_m : p.d_m[which];
        __half* out = sparse ? p.s_out : p.d_out[which];
        const long long st_row = sparse ? p.s_row : p.d_row[which], st_tok = sparse ? p.s_tok : p.d_tok[which];
        const bool vec = st_row == 1 && (st_tok & 7) == 0 && (reinterpret_cast<uintptr_t>(out) & 15u) == 0;
        const bool stored = kSparse ? sparse : which == 0 && p.s_m > 0;
        uint32_t again = 0;
        for (int mb = 0; mb < p.m_blocks; ++mb) {
          const int t = mb * p.inst_m + t_local;
          for (int c = share * 32; c < rows; c += kDecoders * 8) {
            uint32_t r[32];
            tmem_ld32(tmem + (static_cast<uint32_t>(q * 32) << 16) + mb * p.acc_cols + c, r);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            const int left = min(min(rows - c, 32), m_rows - row0 - c);  // what the unit has of these rows
            if (stored && lane_ok && t < p.n && any_nan(r, left)) again |= 1u << mb;
            if (sparse && p.bias != nullptr) {
#pragma unroll
              for (int j = 0; j < 32; ++j) {
                const int row = row0 + c + j;
                const float bv = row < m_rows ? __ldg(p.bias + row) : 0.f;
                r[j] = __float_as_uint(fmaxf(__uint_as_float(r[j]) + bv, 0.f));
              }
            }
            if (!lane_ok || t >= p.n) continue;
            __half* dst = out + static_cast<long long>(row0 + c) * st_row + t * st_tok;
            if (vec) {
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                uint4 pk;
                __half2* h = reinterpret_cast<__half2*>(&pk);
#pragma unroll
                for (int e = 0; e < 4; ++e)
                  h[e] = __floats2half2_rn(__uint_as_float(r[8 * j + 2 * e]), __uint_as_float(r[8 * j + 2 * e + 1]));
                if (8 * j + 8 <= left) {
                  *reinterpret_cast<uint4*>(dst + 8 * j) = pk;
                } else {
                  const __half* hv = reinterpret_cast<const __half*>(&pk);
#pragma unroll
                  for (int e = 0; e < 8; ++e)
                    if (8 * j + e < left) dst[8 * j + e] = hv[e];
                }
              }
            } else {
#pragma unroll
              for (int j = 0; j < 32; ++j)
                if (j < left) dst[j * st_row] = __float2half_rn(__uint_as_float(r[j]));
            }
          }
        }
        if (again != 0) store_again(p, row0, rows, share * 32, t_local, again);
      }
      __syncwarp();
    }
    if (sparse) {
      x_it += k_slots;
      a_it += blocks;
    } else {
      d_it += k_slots;
    }
    // the next unit reuses the accumulator and, if of the other kind, overlays shared memory
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    if (*abort_flag) break;
  }
  __syncthreads();
  if (warp == 1) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(static_cast<uint32_t>(p.tmem_cols))
                 : "memory");
  }
}

// Windows a thread holds twice without spilling registers.
constexpr int kMaxWindows16 = 6, kMaxWindows32 = 4;

struct TilePlan {
  int s_rows, d_rows, kb, windows;
};

int round_up(int v, int to) { return (v + to - 1) / to * to; }

// Rows per unit and columns per block.  A sparse row costs its share of decoder instructions, a
// dense row its bytes; units are sized so that both kinds together occupy the SMs once and end
// together.  Measured on B200 (one SM): about 0.13 ns per stored position of a row plus 16.6 ns per
// row and block of 512 columns; 80 GB/s of dense operand bytes.
bool plan_tile(int m_sparse, int m_dense, int k, int nnz, int index_bits, int sms, int step, int x_slot_bytes,
               TilePlan* out) {
  const double per_row = m_sparse > 0 ? static_cast<double>(nnz) / m_sparse : 0.0;
  const double density = k > 0 ? per_row / k : 0.0;
  const double s_cost = 0.13e-3 * per_row + 0.0166 * ((k + 511) / 512);
  const double d_cost = 2.0 * k / 80e3;
  int s_ctas = sms;
  if (m_dense > 0) {
    const double total = s_cost * m_sparse + d_cost * m_dense;
    s_ctas = m_sparse > 0 ? static_cast<int>(std::lround(sms * s_cost * m_sparse / total)) : 0;
    if (m_sparse > 0) s_ctas = s_ctas < 1 ? 1 : (s_ctas > sms - 1 ? sms - 1 : s_ctas);
  }
  TilePlan pl{step, step, 64, 1};
  if (m_sparse > 0) {
    pl.s_rows = round_up((m_sparse + s_ctas - 1) / s_ctas, step);
    if (pl.s_rows > 128) pl.s_rows = 128;
    s_ctas = (m_sparse + pl.s_rows - 1) / pl.s_rows;
  }
  if (m_dense > 0) {
    const int d_ctas = sms - (s_ctas % sms) > 0 && s_ctas < sms ? sms - s_ctas : sms;
    pl.d_rows = round_up((m_dense + d_ctas - 1) / d_ctas, step);
    if (pl.d_rows > 256) pl.d_rows = round_up((m_dense + 2 * d_ctas - 1) / (2 * d_ctas), step);
    if (pl.d_rows > 256) pl.d_rows = 256;
  }
  if (m_sparse > 0) {
    // Columns per block: as many as two buffers leave room for; U windows of 32 nonzeros have to
    // cover a row's share of a block in almost every case.  Cost of a row and block in instructions:
    // 17 per window and about 110 of its own.
    const int room = kBudget - 2 * x_slot_bytes;
    const int max_u = index_bits == 16 ? kMaxWindows16 : kMaxWindows32;
    double best = 1e30;
    for (int kb = 64; kb <= 512 && kb <= round_up(k, 64); kb += 64) {
      if (2 * (pl.s_rows / 8) * (kb / 64) * 1024 > room) break;
      const double a = density * kb;
      int u = static_cast<int>(std::ceil((a + 1.5 * std::sqrt(a) + 2.0) / 32.0));
      const int rounds = (u + max_u - 1) / max_u;  // windows a row needs in most blocks
      u = u < 1 ? 1 : (u > max_u ? max_u : u);
      const double cost = ((k + kb - 1) / kb) * (17.0 * u * rounds + 110.0);
      if (cost <= best) { best = cost; pl.kb = kb; pl.windows = u; }
    }
    if (best >= 1e30) return false;
    // windows lie inside the arrays as a whole
    while (pl.windows > 1 && 32 * pl.windows > (nnz & ~1)) --pl.windows;
    if (32 * pl.windows > (nnz & ~1)) return false;
  }
  *out = pl;
  return true;
}

template <typename IT, int U, bool kSparse = true>
int launch_tile(const CUtensorMap& mx, const CUtensorMap (&mw)[2], const TileParams& p, int grid, cudaStream_t stream) {
  auto kern = spmm_tile_kernel<IT, U, kSparse>;
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
  return launch_overlapped(kern, dim3(grid), dim3(kThreads), static_cast<size_t>(227 * 1024), stream, mx, mw[0], mw[1], p);
}

template <typename IT>
int dispatch_tile(int windows, const CUtensorMap& mx, const CUtensorMap (&mw)[2], const TileParams& p, int grid,
                  cudaStream_t stream) {
  switch (windows) {
    case 1: return launch_tile<IT, 1>(mx, mw, p, grid, stream);
    case 2: return launch_tile<IT, 2>(mx, mw, p, grid, stream);
    case 3: return launch_tile<IT, 3>(mx, mw, p, grid, stream);
    case 4: return launch_tile<IT, 4>(mx, mw, p, grid, stream);
    default: break;
  }
  if constexpr (sizeof(IT) == 2) {
    if (windows == 5) return launch_tile<IT, 5>(mx, mw, p, grid, stream);
    return launch_tile<IT, 6>(mx, mw, p, grid, stream);
  }
  return IEX_ERR_UNSUPPORTED;
}

// What the outputs and dense matrices of a launch are.
struct DenseArg {
  int m;
  const void* weight;
  void* out;
  int tokens_major;
};

// `copy`: the CSR arrays are those of dense[0], which is their dense copy, and not of a matrix that is decoded.
int tile_launch(bool copy, int m_sparse, int k, int n, int nnz, const int32_t* row_offsets, const void* cols, int index_bits,
                const void* values, const float* bias, void* out_sparse, int sparse_tokens_major,
                const DenseArg (&dense)[2], const void* x, int x_tokens_major, void* stream) {
  const int m_dense = dense[0].m + dense[1].m;
  if (m_sparse < 0 || dense[0].m < 0 || dense[1].m < 0 || k < 0 || n < 0 || nnz < 0) return IEX_ERR_BAD_ARG;
  if (index_bits != 16 && index_bits != 32) return IEX_ERR_BAD_ARG;
  if ((m_sparse == 0 && m_dense == 0) || n == 0) return IEX_OK;
  if (copy && dense[0].m > 0 && (!row_offsets || !cols || !values)) return IEX_ERR_BAD_ARG;
  if (!x || (m_sparse > 0 && (!row_offsets || !out_sparse || (nnz > 0 && (!cols || !values))))) return IEX_ERR_BAD_ARG;
  for (const auto& d : dense)
    if (d.m > 0 && (!d.weight || !d.out)) return IEX_ERR_BAD_ARG;
  if (n > 256 || k == 0 || (x_tokens_major ? k : n) % 8 != 0 || (m_dense > 0 && k % 8 != 0)) return IEX_ERR_UNSUPPORTED;
  if (index_bits == 16 && k > 65024) return IEX_ERR_UNSUPPORTED;  // 0xffff marks padding in every block
  if (!aligned16(x) || (dense[0].m > 0 && !aligned16(dense[0].weight)) || (dense[1].m > 0 && !aligned16(dense[1].weight)))
    return IEX_ERR_UNSUPPORTED;
  if (m_sparse > 0 && ((reinterpret_cast<uintptr_t>(values) & 3u) != 0 ||
                       (reinterpret_cast<uintptr_t>(cols) & static_cast<uintptr_t>(index_bits / 4 - 1)) != 0))
    return IEX_ERR_UNSUPPORTED;  // pairs of nonzeros are loaded together
  TileParams p{};
  p.inst_m = n <= 64 ? 64 : 128;
  p.m_blocks = n <= 128 ? 1 : 2;
  const int step = p.inst_m == 64 ? 8 : 16;
  const int x_slot = p.inst_m * p.m_blocks * 128;
  const int sms = sm_count();
  TilePlan pl{};
  if (!plan_tile(m_sparse, m_dense, k, nnz, index_bits, sms, step, x_slot, &pl)) return IEX_ERR_UNSUPPORTED;
  p.s_rows = pl.s_rows;
  p.s_tiles = m_sparse > 0 ? (m_sparse + pl.s_rows - 1) / pl.s_rows : 0;
  p.s_m = m_sparse;
  p.s_nnz = nnz;
  p.row_offsets = row_offsets;
  p.cols = cols;
  p.values = static_cast<const __half*>(values);
  p.bias = bias;
  p.s_out = static_cast<__half*>(out_sparse);
  p.s_row = sparse_tokens_major ? 1 : n;
  p.s_tok = sparse_tokens_major ? m_sparse : 1;
  p.d_rows = pl.d_rows;
  for (int i = 0; i < 2; ++i) {
    p.d_tiles[i] = (dense[i].m + pl.d_rows - 1) / pl.d_rows;
    p.d_m[i] = dense[i].m;
    p.d_out[i] = static_cast<__half*>(dense[i].out);
    p.d_row[i] = dense[i].tokens_major ? 1 : n;
    p.d_tok[i] = dense[i].tokens_major ? dense[i].m : 1;
  }
  if (copy) {  // where store_again finds its outputs
    p.s_m = dense[0].m;
    p.s_out = p.d_out[0];
    p.s_row = p.d_row[0];
    p.s_tok = p.d_tok[0];
  }
  p.k = k;
  p.n = n;
  p.x_mn = x_tokens_major ? 0 : 1;
  p.terms.row_offsets = row_offsets;
  p.terms.cols = cols;
  p.terms.values = p.values;
  p.terms.dense = static_cast<const __half*>(x);
  p.terms.dense_c = p.x_mn ? n : 1;
  p.terms.dense_t = p.x_mn ? 1 : k;
  p.terms.rows = copy ? dense[0].m : m_sparse;
  p.terms.columns = n;
  p.terms.index_bits = index_bits;
  p.kb = pl.kb;
  const int widest = (m_sparse > 0 && p.s_rows > p.d_rows) || m_dense == 0 ? p.s_rows : p.d_rows;
  p.acc_cols = round_up(widest, 32);
  p.tmem_cols = 32;
  while (p.tmem_cols < p.acc_cols * p.m_blocks) p.tmem_cols <<= 1;
  p.ahead = 2 * 32 * pl.windows;
  p.status = status_word();
  p.x_slots = 1;
  if (m_sparse > 0) {
    const int left = kBudget - 2 * (p.s_rows / 8) * (p.kb / 64) * 1024;
    p.x_slots = left / x_slot > kMaxXSlots ? kMaxXSlots : left / x_slot;
    if (p.x_slots < 2) return IEX_ERR_UNSUPPORTED;
  }
  p.stages = 1;
  if (m_dense > 0) {
    p.stages = kBudget / (x_slot + p.d_rows * 128);
    p.stages = p.stages > kMaxStages ? kMaxStages : p.stages;
    if (p.stages < 2) return IEX_ERR_UNSUPPORTED;
  }
  CUtensorMap mx, mw[2];
  int st = p.x_mn ? make_map_f16(&mx, x, k, n, n, 64, 64, true)
                  : make_map_f16(&mx, x, n, k, k, p.inst_m * p.m_blocks, 64, true);
  for (int i = 0; i < 2; ++i) {
    if (st == IEX_OK && dense[i].m > 0) st = make_map_f16(&mw[i], dense[i].weight, dense[i].m, k, k, p.d_rows, 64, true);
    if (dense[i].m == 0) mw[i] = mx;
  }
  if (st != IEX_OK) return st;
  const int units = p.s_tiles + p.d_tiles[0] + p.d_tiles[1];
  const int grid = units < sms ? units : sms;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (m_sparse == 0) return launch_tile<uint16_t, 1, false>(mx, mw, p, grid, s);
  if (index_bits == 16) return dispatch_tile<uint16_t>(pl.windows, mx, mw, p, grid, s);
  return dispatch_tile<int>(pl.windows, mx, mw, p, grid, s);
}

}  // namespace
}  // namespace tc
}  // namespace iex

extern "C" int iex_spmm_linear_f16_tile(int m_sparse, int m_dense, int k, int n, int nnz, const int32_t* row_offsets,
                                        const void* column_indices, int index_bits, const void* values,
                                        const void* weight, const void* x, int x_tokens_major, const float* bias,
                                        void* out_sparse, int sparse_tokens_major, void* out_dense,
                                        int dense_tokens_major, void* stream) {
  const iex::tc::DenseArg dense[2] = {{m_dense, weight, out_dense, dense_tokens_major}, {0, nullptr, nullptr, 0}};
  return iex::tc::tile_launch(false, m_sparse, k, n, nnz, row_offsets, column_indices, index_bits, values, bias, out_sparse,
                              sparse_tokens_major, dense, x, x_tokens_major, stream);
}

extern "C" int iex_linear_pair_f16_csr(int m0, int m1, int k, int n, const void* weight0, const int32_t* row_offsets,
                                       const void* column_indices, int index_bits, const void* values, const void* weight1,
                                       const void* x, int x_tokens_major, void* out0, int tokens_major0, void* out1,
                                       int tokens_major1, void* stream) {
  const iex::tc::DenseArg dense[2] = {{m0, weight0, out0, tokens_major0}, {m1, weight1, out1, tokens_major1}};
  return iex::tc::tile_launch(row_offsets != nullptr, 0, k, n, 0, row_offsets, column_indices, index_bits, values, nullptr, nullptr, 0, dense, x,
                              x_tokens_major, stream);
}

extern "C" int iex_linear_pair_f16(int m0, int m1, int k, int n, const void* weight0, const void* weight1, const void* x,
                                   int x_tokens_major, void* out0, int tokens_major0, void* out1, int tokens_major1,
                                   void* stream) {
  return iex_linear_pair_f16_csr(m0, m1, k, n, weight0, nullptr, nullptr, 16, nullptr, weight1, x, x_tokens_major, out0,
                                 tokens_major0, out1, tokens_major1, stream);
}
