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
//   warps 2-17   sparse units: CSR decoders.  Each owns rows of the unit.  Block by block (kb columns,
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
// row in rounds of dependent steps (29 thread instructions per nonzero against about 12 here).
//
// Row groups of 8 hold their 64-column atoms next to each other (descriptor stride kb / 64 KB), so
// that a column's offset inside a row group is two bit fields of the column and no multiplication.
//
// Every mbarrier wait is bounded, as in tc_fused.cu.
#include <cuda.h>

#include <cmath>
#include <mutex>

#include "common.cuh"
#include "tc_ptx.cuh"

namespace iex {
namespace tc {

int make_map_f16(CUtensorMap* map, const void* base, long long rows, long long cols, long long ld, int box_rows,
                 int box_cols, bool swizzle);  // tc_fused.cu

namespace {

constexpr int kDecoders = 16;
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
  // dense units
  int d_tiles, d_rows, d_m;
  __half* d_out;
  long long d_row, d_tok;
  // shared
  int k, n;
  int x_mn;            // X stored [k, n] (tokens contiguous), else [n, k]
  int inst_m;          // tokens per MMA: 64 or 128
  int m_blocks;        // 1 or 2 of them
  int kb;              // columns per sparse block, a multiple of 64 up to 512
  int x_slots, stages;
  int acc_cols, tmem_cols;
  int ahead;           // nonzeros of L2 prefetch distance
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

// U pairs of a lane as loaded, the columns in the matrix's index type.
template <typename IT, int U> struct Window;
template <int U> struct Window<uint16_t, U> { uint32_t v[U], c[U]; };
template <int U> struct Window<int, U> { uint32_t v[U]; int2 c[U]; };

// Requests positions [base, base + 64 U) of one row; pairs that start at or past `end` hold an
// index no block contains.
template <typename IT, int U>
__device__ __forceinline__ void load_window(Window<IT, U>& w, const __half* __restrict__ values,
                                            const IT* __restrict__ cols, int base, int end, int nnz, int lane) {
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const int p = base + 64 * u + 2 * lane;
    if constexpr (sizeof(IT) == 2) w.c[u] = 0xffffffffu; else w.c[u] = make_int2(-1, -1);
    w.v[u] = 0u;
    if (p < end) {
      if (p + 1 < nnz) {
        w.v[u] = __ldg(reinterpret_cast<const uint32_t*>(values + p));
        if constexpr (sizeof(IT) == 2) w.c[u] = __ldg(reinterpret_cast<const uint32_t*>(cols + p));
        else w.c[u] = __ldg(reinterpret_cast<const int2*>(cols + p));
      } else {  // last nonzero of the arrays
        w.v[u] = __half_as_ushort(__ldg(values + p));
        if constexpr (sizeof(IT) == 2) w.c[u] = 0xffff0000u | __ldg(cols + p);
        else w.c[u] = make_int2(__ldg(cols + p), -1);
      }
    }
  }
}
// Both columns of pair u relative to the block's first column, 16 bits each; anything outside the
// block is at least kb (columns below the block only occur before `cur` and are excluded there).
template <int U>
__device__ __forceinline__ uint32_t relative(const Window<uint16_t, U>& w, int u, uint32_t c0, bool skip_first) {
  uint32_t c = w.c[u];
  if (skip_first) c = (c & 0xffff0000u) | (c >> 16);  // keeps the packed subtraction free of a borrow
  return c - (c0 | (c0 << 16));
}
template <int U>
__device__ __forceinline__ uint32_t relative(const Window<int, U>& w, int u, uint32_t c0, bool) {
  const uint32_t a = min(static_cast<uint32_t>(w.c[u].x) - c0, 0xffffu);
  const uint32_t b = min(static_cast<uint32_t>(w.c[u].y) - c0, 0xffffu);
  return a | (b << 16);
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

template <typename IT, int U>
__global__ void __launch_bounds__(kThreads, 1)
spmm_tile_kernel(const __grid_constant__ CUtensorMap map_x_s, const __grid_constant__ CUtensorMap map_w,
                 const TileParams p) {
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
  const int units = p.s_tiles + p.d_tiles;
  uint32_t x_it = 0, d_it = 0, a_it = 0;  // slots / stages / blocks used so far (each role counts alike)
  uint32_t unit_it = 0;

  for (int u = blockIdx.x; u < units; u += gridDim.x, ++unit_it) {
    const bool sparse = u < p.s_tiles;
    const int rows = sparse ? p.s_rows : p.d_rows;
    const int row0 = (sparse ? u : u - p.s_tiles) * rows;
    if (warp == 0) {
      // ---------------------------------------------------------------- TMA producer
      if (elect_one()) {
        const int m_atoms = p.inst_m * p.m_blocks / 64;
        auto load_x = [&](uint32_t dst, uint32_t full, int ks) {
          if (p.x_mn) {
            for (int j = 0; j < m_atoms; ++j) tma_load_2d(dst + j * 8192u, &map_x_s, full, j * 64, ks * 64);
          } else {
            tma_load_2d(dst, &map_x_s, full, ks * 64, 0);
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
            tma_load_2d(dst + x_bytes, &map_w, d_full(s), ks * 64, row0);
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
        const int nrows = (rows - w + kDecoders - 1) / kDecoders;  // this warp's rows: w, w + 16, ...
        // lane i holds the position and the end of the warp's row i
        int cur_l = 0, end_l = 0;
        if (lane < nrows) {
          const int r = row0 + w + kDecoders * lane;
          if (r < p.s_m) {
            cur_l = __ldg(p.row_offsets + r);
            end_l = __ldg(p.row_offsets + r + 1);
          }
        }
        auto prefetch = [&](int from, int end) {  // eight 128-byte lines of values and of indices
          const int l8 = lane & 7;
          if (lane < 8) {
            const int q = from + l8 * 64;
            if (q < end && 64 * l8 < p.ahead) asm volatile("prefetch.global.L2 [%0];" ::"l"(p.values + q));
          } else if (lane < 8 + 8 * static_cast<int>(sizeof(IT)) / 2) {
            constexpr int kPer = 128 / sizeof(IT);
            const int q = from + (lane - 8) * kPer;
            if (q < end && kPer * (lane - 8) < p.ahead) asm volatile("prefetch.global.L2 [%0];" ::"l"(cols + q));
          }
        };
        Window<IT, U> win, next;
        if (nrows > 0) {
          for (int i = 0; i < nrows; ++i)
            prefetch(__shfl_sync(0xffffffffu, cur_l, i), __shfl_sync(0xffffffffu, end_l, i));
          const int c = __shfl_sync(0xffffffffu, cur_l, 0), e = __shfl_sync(0xffffffffu, end_l, 0);
          load_window<IT, U>(win, p.values, cols, c & ~1, e, p.s_nnz, lane);
        }
        for (int b = 0; b < blocks; ++b) {
          const uint32_t ab = a_it + b;
          const uint32_t buf = base + (ab & 1u) * block_bytes;
          const uint32_t c0 = static_cast<uint32_t>(b * p.kb);
          if (!mbar_wait(a_empty(ab & 1u), ((ab >> 1) & 1u) ^ 1u, abort_flag, p.status, 32)) { ok = false; break; }
          // clear this warp's rows: 8 lanes per 128-byte row of an atom, four atoms at a time
          for (int i = 0; i < nrows; ++i) {
            const uint32_t r = w + kDecoders * i;
            const uint32_t dst = buf + (r >> 3) * atoms * 1024u + (r & 7u) * 128u + (lane & 7) * 16u;
            for (uint32_t j = lane >> 3; j < atoms; j += 4)
              asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(dst + j * 1024u), "r"(0u) : "memory");
          }
          __syncwarp();
          for (int i = 0; i < nrows; ++i) {
            int cur = __shfl_sync(0xffffffffu, cur_l, i);
            const int end = __shfl_sync(0xffffffffu, end_l, i);
            const int ni = i + 1 < nrows ? i + 1 : 0;
            const bool more_items = i + 1 < nrows || b + 1 < blocks;
            if (nrows > 1 && more_items) {  // the next row's window travels while this one is written
              const int nc = __shfl_sync(0xffffffffu, cur_l, ni), ne = __shfl_sync(0xffffffffu, end_l, ni);
              load_window<IT, U>(next, p.values, cols, nc & ~1, ne, p.s_nnz, lane);
            }
            prefetch(cur + p.ahead, end);
            const uint32_t r = w + kDecoders * i;
            const uint32_t row_base = buf + (r >> 3) * atoms * 1024u + (r & 7u) * 128u;
            const uint32_t sw = (r & 7u) << 4, sw2 = sw | (sw << 16);
            const uint32_t kb = static_cast<uint32_t>(p.kb);
            for (;;) {
              const int wbase = cur & ~1;
              uint32_t rel[U];
              bool v0[U], v1[U];
              int cnt = 0;
#pragma unroll
              for (int q = 0; q < U; ++q) {
                const int pos = wbase + 64 * q + 2 * lane;
                rel[q] = relative<U>(win, q, c0, q == 0 && pos < cur);
                v0[q] = (rel[q] & 0xffffu) < kb && pos < end && (q > 0 || pos >= cur);
                v1[q] = (rel[q] >> 16) < kb && pos + 1 < end;
                cnt += __popc(__ballot_sync(0xffffffffu, v0[q])) + __popc(__ballot_sync(0xffffffffu, v1[q]));
              }
              cur += cnt;
              const bool again = cur == wbase + 64 * U && cur < end;  // the whole window fell into the block
              if (!again) {
                if (lane == i) cur_l = cur;
                if (nrows == 1 && more_items) load_window<IT, U>(next, p.values, cols, cur & ~1, end, p.s_nnz, lane);
              }
#pragma unroll
              for (int q = 0; q < U; ++q) {
                // offset inside the row group: 64-column atom (bits 6-8 of the column) and swizzled byte
                const uint32_t off = ((rel[q] << 4) & 0x1c001c00u) | (((rel[q] << 1) & 0x007e007eu) ^ sw2);
                if (v0[q])
                  asm volatile("st.shared.u16 [%0], %1;" ::"r"(row_base + (off & 0xffffu)),
                               "h"(static_cast<uint16_t>(win.v[q])) : "memory");
                if (v1[q])
                  asm volatile("st.shared.u16 [%0], %1;" ::"r"(row_base + (off >> 16)),
                               "h"(static_cast<uint16_t>(win.v[q] >> 16)) : "memory");
              }
              if (!again) break;
              load_window<IT, U>(win, p.values, cols, cur, end, p.s_nnz, lane);
            }
            win = next;
          }
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          __syncwarp();
          if (lane == 0) mbar_arrive(a_full(ab & 1u));
        }
      }
      // ---------------------------------------------------------------- read-out
      if (ok && mbar_wait(acc_full, unit_it & 1u, abort_flag, p.status, 64)) {
        tcgen05_fence_after();
        const int q = warp & 3, share = w >> 2;  // tensor-memory quarter; four warps split its columns
        const int t_local = p.inst_m == 64 ? q * 16 + lane : q * 32 + lane;
        const bool lane_ok = p.inst_m == 128 || lane < 16;
        const int m_rows = sparse ? p.s_m : p.d_m;
        __half* out = sparse ? p.s_out : p.d_out;
        const long long st_row = sparse ? p.s_row : p.d_row, st_tok = sparse ? p.s_tok : p.d_tok;
        const bool vec = st_row == 1 && (st_tok & 7) == 0 && (reinterpret_cast<uintptr_t>(out) & 15u) == 0;
        for (int mb = 0; mb < p.m_blocks; ++mb) {
          const int t = mb * p.inst_m + t_local;
          for (int c = share * 32; c < rows; c += 128) {
            uint32_t r[32];
            tmem_ld32(tmem + (static_cast<uint32_t>(q * 32) << 16) + mb * p.acc_cols + c, r);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            if (sparse && p.bias != nullptr) {
#pragma unroll
              for (int j = 0; j < 32; ++j) {
                const int row = row0 + c + j;
                const float bv = row < m_rows ? __ldg(p.bias + row) : 0.f;
                r[j] = __float_as_uint(fmaxf(__uint_as_float(r[j]) + bv, 0.f));
              }
            }
            if (!lane_ok || t >= p.n) continue;
            const int left = min(min(rows - c, 32), m_rows - row0 - c);
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

struct TilePlan {
  int s_rows, d_rows, kb, windows;
};

int round_up(int v, int to) { return (v + to - 1) / to * to; }

// Rows per unit and columns per block.  A sparse row costs its share of decoder instructions, a
// dense row its bytes; units are sized so that both kinds together occupy the SMs once and end
// together.  Measured on B200 (one SM): about 0.9 ns per stored position of a row plus 16 ns per
// row and block; 95 GB/s of dense operand bytes.
bool plan_tile(int m_sparse, int m_dense, int k, int n, int nnz, int sms, int step, int x_slot_bytes, TilePlan* out) {
  const double per_row = m_sparse > 0 ? static_cast<double>(nnz) / m_sparse : 0.0;
  const double density = k > 0 ? per_row / k : 0.0;
  const double s_cost = 0.9e-3 * per_row + 0.016 * ((k + 447) / 448);
  const double d_cost = 2.0 * k / 95e3;
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
    // Columns per block: as many as two buffers leave room for; U windows of 64 nonzeros have to
    // cover a row's share of a block in almost every case.  Cost of a row and block in instructions:
    // 17 per window and about 45 of its own.
    const int room = kBudget - 2 * x_slot_bytes;
    double best = 1e30;
    for (int kb = 64; kb <= 512 && kb <= round_up(k, 64); kb += 64) {
      if (2 * (pl.s_rows / 8) * (kb / 64) * 1024 > room) break;
      const double a = density * kb;
      int u = static_cast<int>(std::ceil((a + 1.5 * std::sqrt(a) + 2.0) / 64.0));
      u = u < 1 ? 1 : (u > 5 ? 5 : u);
      const double cost = ((k + kb - 1) / kb) * (17.0 * u + 45.0) * std::fmax(1.0, a / (64.0 * u));
      if (cost <= best) { best = cost; pl.kb = kb; pl.windows = u; }
    }
    if (best >= 1e30) return false;
  }
  *out = pl;
  return true;
}

template <typename IT, int U>
int launch_tile(const CUtensorMap& mx, const CUtensorMap& mw, const TileParams& p, int grid, cudaStream_t stream) {
  auto kern = spmm_tile_kernel<IT, U>;
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
  return launch_overlapped(kern, dim3(grid), dim3(kThreads), static_cast<size_t>(227 * 1024), stream, mx, mw, p);
}

template <typename IT>
int dispatch_tile(int windows, const CUtensorMap& mx, const CUtensorMap& mw, const TileParams& p, int grid,
                  cudaStream_t stream) {
  switch (windows) {
    case 1: return launch_tile<IT, 1>(mx, mw, p, grid, stream);
    case 2: return launch_tile<IT, 2>(mx, mw, p, grid, stream);
    case 3: return launch_tile<IT, 3>(mx, mw, p, grid, stream);
    case 4: return launch_tile<IT, 4>(mx, mw, p, grid, stream);
    default: return launch_tile<IT, 5>(mx, mw, p, grid, stream);
  }
}

}  // namespace
}  // namespace tc
}  // namespace iex

extern "C" int iex_spmm_linear_f16_tile(int m_sparse, int m_dense, int k, int n, int nnz, const int32_t* row_offsets,
                                        const void* column_indices, int index_bits, const void* values,
                                        const void* weight, const void* x, int x_tokens_major, const float* bias,
                                        void* out_sparse, int sparse_tokens_major, void* out_dense,
                                        int dense_tokens_major, void* stream) {
  using namespace iex;
  using namespace iex::tc;
  if (m_sparse < 0 || m_dense < 0 || k < 0 || n < 0 || nnz < 0) return IEX_ERR_BAD_ARG;
  if (index_bits != 16 && index_bits != 32) return IEX_ERR_BAD_ARG;
  if ((m_sparse == 0 && m_dense == 0) || n == 0) return IEX_OK;
  if (!x || (m_sparse > 0 && (!row_offsets || !out_sparse || (nnz > 0 && (!column_indices || !values)))))
    return IEX_ERR_BAD_ARG;
  if (m_dense > 0 && (!weight || !out_dense)) return IEX_ERR_BAD_ARG;
  if (n > 256 || k == 0 || (x_tokens_major ? k : n) % 8 != 0 || (m_dense > 0 && k % 8 != 0)) return IEX_ERR_UNSUPPORTED;
  if (index_bits == 16 && k > 65024) return IEX_ERR_UNSUPPORTED;  // 0xffff marks padding in every block
  if (!aligned16(x) || (m_dense > 0 && !aligned16(weight))) return IEX_ERR_UNSUPPORTED;
  if ((reinterpret_cast<uintptr_t>(values) & 3u) != 0 ||
      (reinterpret_cast<uintptr_t>(column_indices) & static_cast<uintptr_t>(index_bits / 4 - 1)) != 0)
    return IEX_ERR_UNSUPPORTED;  // pairs of nonzeros are loaded together
  TileParams p{};
  p.inst_m = n <= 64 ? 64 : 128;
  p.m_blocks = n <= 128 ? 1 : 2;
  const int step = p.inst_m == 64 ? 8 : 16;
  const int x_slot = p.inst_m * p.m_blocks * 128;
  const int sms = sm_count();
  TilePlan pl{};
  if (!plan_tile(m_sparse, m_dense, k, n, nnz, sms, step, x_slot, &pl)) return IEX_ERR_UNSUPPORTED;
  p.s_rows = pl.s_rows;
  p.s_tiles = m_sparse > 0 ? (m_sparse + pl.s_rows - 1) / pl.s_rows : 0;
  p.s_m = m_sparse;
  p.s_nnz = nnz;
  p.row_offsets = row_offsets;
  p.cols = column_indices;
  p.values = static_cast<const __half*>(values);
  p.bias = bias;
  p.s_out = static_cast<__half*>(out_sparse);
  p.s_row = sparse_tokens_major ? 1 : n;
  p.s_tok = sparse_tokens_major ? m_sparse : 1;
  p.d_rows = pl.d_rows;
  p.d_tiles = m_dense > 0 ? (m_dense + pl.d_rows - 1) / pl.d_rows : 0;
  p.d_m = m_dense;
  p.d_out = static_cast<__half*>(out_dense);
  p.d_row = dense_tokens_major ? 1 : n;
  p.d_tok = dense_tokens_major ? m_dense : 1;
  p.k = k;
  p.n = n;
  p.x_mn = x_tokens_major ? 0 : 1;
  p.kb = pl.kb;
  const int widest = (m_sparse > 0 && p.s_rows > p.d_rows) || m_dense == 0 ? p.s_rows : p.d_rows;
  p.acc_cols = round_up(widest, 32);
  p.tmem_cols = 32;
  while (p.tmem_cols < p.acc_cols * p.m_blocks) p.tmem_cols <<= 1;
  p.ahead = 2 * 64 * pl.windows < 512 ? 2 * 64 * pl.windows : 512;
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
  CUtensorMap mx, mw;
  int st = p.x_mn ? make_map_f16(&mx, x, k, n, n, 64, 64, true)
                  : make_map_f16(&mx, x, n, k, k, p.inst_m * p.m_blocks, 64, true);
  if (st == IEX_OK && m_dense > 0) st = make_map_f16(&mw, weight, m_dense, k, k, p.d_rows, 64, true);
  if (st != IEX_OK) return st;
  if (m_dense == 0) mw = mx;
  const int units = p.s_tiles + p.d_tiles;
  const int grid = units < sms ? units : sms;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (index_bits == 16) return dispatch_tile<uint16_t>(pl.windows, mx, mw, p, grid, s);
  return dispatch_tile<int>(pl.windows, mx, mw, p, grid, s);
}
