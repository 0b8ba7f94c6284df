// CSR SpMM on CUDA cores with the dense operand in shared memory (sm_100a):
//   out[z, r, :] = sum_p values[p] * dense[z, col[p], :].
//
// spmm_simt.cu gathers a row of `dense` from L2 for every nonzero and gives a row of A to one group of
// lanes: with a few thousand row groups in all it is bound by the walk along the longest row, an L2 latency
// for every 8 to 16 nonzeros (1024 x 1024 at 90 % x 256 in fp32: 260 nonzeros in the longest row, 16.5 us).
//
// Here a CTA keeps a slice (128, 64 or 32 bytes) of every row of `dense`, brought in once by TMA, and walks its share of
// the rows against it: the gathers take a shared-memory latency instead of an L2 one, and L2 delivers 19 MB
// instead of 107 MB in that example.  A warp works on 1 to 8 rows at once that follow each other in the order by length, so they are
// about as long as each other and the loops are uniform; a nonzero that one of them has no counterpart for is replaced
// by zero times a row of zeros.  Nonzeros stream through a ring of windows per warp.  As in
// spmm_simt.cu every output is summed by one lane, in storage order: the same bits.
//
// Bound by what shared memory returns to registers (128 bytes a cycle): W bytes of columns for a nonzero, and
// its value and column for each lane of the row, which cost as much again.  So a lane takes 8 bytes of
// columns rather than 4 where there are rows enough; 16 bytes left too few bunches of rows for the warps.
//   fp32  1024 x 1024 at 90 % x 256: 16.5 -> 10.3 us    1531 x 1177 at 85 % x 100: 21.8 -> 15.1 us
//   fp16  1024 x 1024 at 90 % x 256: 21.1 -> 9.4 us     512 x 512 at 50 % x 128: 31.7 -> 8.6 us
// Of the 10.3 us 2 pass before the first product (launch, the slice, the chain row number - offsets - nonzeros).
// Splitting rows between warps and lanes instead, for balance, was slower (11.9 us) and changed the bits.
#include <algorithm>
#include <mutex>

#include <cuda.h>

#include "common.cuh"
#include "tc_ptx.cuh"

namespace iex {
namespace tc {

int make_map_slice(CUtensorMap* map, bool half, const void* base, long long rows, long long cols, int box_rows,
                   int box_cols);  // tc_fused.cu
int* status_word();                // tc_fused.cu

}  // namespace tc

namespace {

using namespace tc;

constexpr int kWarps = 16;
constexpr int kStages = 2;               // windows of nonzeros a warp keeps in shared memory
constexpr int kBoxRows = 64;             // rows of the dense operand in one TMA box
constexpr int kSmemBytes = 227 * 1024;   // of a CTA, all uses

struct Params {
  int m, k, n, nnz;
  int tiles, units, groups;
  long long values_batch_stride;
  const int* row_indices;
  const int* row_offsets;
  const void* values;
  const void* cols;
  const void* dense;
  const float* bias;
  void* out;
  int accumulate;
  int* status;
};

__device__ __forceinline__ uint4 lds128(uint32_t at) {
  uint4 v;
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(at));
  return v;
}
// Nonzeros of a warp's window, all rows of it together.  Wide slices leave room for less.
template <typename VT, typename IT, int W>
constexpr int window() { return (sizeof(VT) == 4 || sizeof(IT) == 4 ? 64 : 128) * (W == 128 ? 2 : 4); }
// Bytes of a window in the ring: a header and the nonzeros of each row, 16 bytes apart in banks.
template <typename VT, typename IT, int W, int B>
constexpr int stage_bytes() { return window<VT, IT, W>() * static_cast<int>(sizeof(VT) + sizeof(IT)) + 32 * (32 * B / W); }

template <int B> struct LaneWord;
template <> struct LaneWord<4> { uint32_t x[1]; };
template <> struct LaneWord<8> { uint32_t x[2]; };
template <> struct LaneWord<16> { uint32_t x[4]; };
template <int B>
__device__ __forceinline__ LaneWord<B> lds(uint32_t at) {
  LaneWord<B> v;
  if constexpr (B == 4) asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v.x[0]) : "r"(at));
  if constexpr (B == 8) asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(v.x[0]), "=r"(v.x[1]) : "r"(at));
  if constexpr (B == 16)
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x[0]), "=r"(v.x[1]), "=r"(v.x[2]), "=r"(v.x[3]) : "r"(at));
  return v;
}

// W    bytes of a slice's row
// B    bytes of columns of a lane: W / B lanes have a row of A, and a warp works on 32 * B / W rows at once
// VDN  rows of `dense` are multiples of 16 bytes: the slice is filled by TMA
template <typename VT, typename IT, int W, int B, bool VDN>
__global__ void __launch_bounds__(kWarps * 32)
spmm_slice_kernel(const __grid_constant__ CUtensorMap map, const __grid_constant__ Params q) {
  constexpr int kThreads = kWarps * 32;
  constexpr int L = W / B, S = 32 / L;
  constexpr uint32_t kRow = W;
  constexpr int CPL = B / sizeof(VT);               // columns of a lane
  constexpr int kWidth = L * CPL;                   // columns of a slice
  constexpr int VN = 16 / sizeof(VT);               // nonzeros of a pack
  constexpr int kWin = window<VT, IT, W>() / S;        // nonzeros of a row in a window
  constexpr int kPacks = kWin / VN;
  constexpr int kVP = kWin * sizeof(VT) / 16, kCP = kWin * sizeof(IT) / 16;  // 16-byte pieces: values, columns
  constexpr uint32_t kSub = kWin * (sizeof(VT) + sizeof(IT)) + 16;
  constexpr uint32_t kStage = stage_bytes<VT, IT, W, B>();
  constexpr int kIdx = sizeof(IT) * VN / 16;        // loads for the columns of a pack
  extern __shared__ __align__(128) uint8_t slice_smem[];
  __shared__ __align__(8) uint64_t s_bar;
  __shared__ int s_abort;

  const int lane = threadIdx.x & 31, sub = lane / L, sl = lane % L, warp = threadIdx.x >> 5;
  const uint32_t slice = smem_u32(slice_smem), bar = smem_u32(&s_bar);
  const int boxes = (q.k + kBoxRows - 1) / kBoxRows;
  const uint32_t mine = slice + sl * B;
  const uint32_t zero_row = mine + boxes * kBoxRows * kRow;  // what stands in for a nonzero that is not the row's
  const uint32_t ring = slice + boxes * kBoxRows * kRow + 128u + warp * kStages * kStage;
  if (threadIdx.x < 32) reinterpret_cast<uint32_t*>(slice_smem + boxes * kBoxRows * kRow)[threadIdx.x] = 0;
  if (VDN && threadIdx.x == 0) {
    mbar_init(bar, 1);
    s_abort = 0;
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  grid_dependency_wait();  // the kernel before this one may have written what is read below
  grid_launch_dependents();
  const IT* cols = static_cast<const IT*>(q.cols);
  const int bunches = (q.m + S - 1) / S;

  uint32_t phase = 0;
  for (int unit = blockIdx.x; unit < q.units; unit += gridDim.x, phase ^= 1u) {
    const int item = unit / q.groups, group = unit - item * q.groups;
    const int z = item / q.tiles, c0 = (item - z * q.tiles) * kWidth;
    const int width = min(kWidth, q.n - c0);
    const VT* vals = static_cast<const VT*>(q.values) + static_cast<size_t>(z) * static_cast<size_t>(q.values_batch_stride);
    __syncthreads();  // the unit before this one is done with
    if (VDN && warp == kWarps - 1 && elect_one()) {
      mbar_arrive_expect_tx(bar, boxes * kBoxRows * kRow);
      for (int i = 0; i < boxes; ++i)
        tma_load_2d(slice + i * kBoxRows * kRow, &map, bar, c0, z * q.k + i * kBoxRows);
    }
    __syncwarp();

    // This CTA's rows are every groups-th bunch of S rows of the order by length, this warp's every kWarps-th of
    // those, to and fro, so that every warp has long ones and short ones.
    const int rounds = (bunches - group + q.groups * kWarps - 1) / (q.groups * kWarps);
    auto row_at = [&](int t) {
      const int j = t * kWarps + ((t & 1) ? kWarps - 1 - warp : warp);
      const long long slot = (group + static_cast<long long>(j) * q.groups) * S + sub;
      return t < rounds && slot < q.m ? __ldg(q.row_indices + slot) : -1;
    };
    // The stream of windows: the row at hand, the one after it, and the number of the one after that.
    int gt = 0, gw = 0, gr = row_at(0), nr = row_at(1), nnr = row_at(2);
    int gbeg = 0, gend = 0, nbeg = 0, nend = 0;
    if (gr >= 0) { gbeg = __ldg(q.row_offsets + gr); gend = __ldg(q.row_offsets + gr + 1); }
    if (nr >= 0) { nbeg = __ldg(q.row_offsets + nr); nend = __ldg(q.row_offsets + nr + 1); }
    auto windows = [&](int beg, int end) {
      int w = max((end - (beg & ~(VN - 1)) + kWin - 1) / kWin, 1);
      if constexpr (S > 1) w = __reduce_max_sync(0xffffffffu, w);
      return w;
    };
    int gn = windows(gbeg, gend);
    auto produce = [&](uint32_t stage) {
      if (gt < rounds) {
        const int base = (gbeg & ~(VN - 1)) + gw * kWin;
        const uint32_t to = stage + S * 16u + sub * kSub;
#pragma unroll
        for (int i0 = 0; i0 < kVP + kCP; i0 += L) {
          const int i = i0 + sl;
          if ((kVP + kCP) % L != 0 && i >= kVP + kCP) break;
          const bool val = i < kVP;
          const int e = base + (val ? i * VN : (i - kVP) * (16 / static_cast<int>(sizeof(IT))));
          const int size = val ? static_cast<int>(sizeof(VT)) : static_cast<int>(sizeof(IT));
          // past the arrays: zeros (the minimum first: the bytes that are left can be more than an int holds)
          const int rest = e < gend ? min(q.nnz - e, 16 / size) * size : 0;
          const char* src = val ? reinterpret_cast<const char*>(vals + e) : reinterpret_cast<const char*>(cols + e);
          asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(to + i * 16u),
                       "l"(rest > 0 ? src : reinterpret_cast<const char*>(cols)), "r"(rest)
                       : "memory");
        }
        ++gw;
        if (sl == 0)
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(stage + sub * 16u), "r"(gr), "r"(gbeg), "r"(gend),
                       "r"(gw == gn ? -gw : gw)
                       : "memory");
        if (gw == gn) {
          gw = 0;
          ++gt;
          gr = nr; gbeg = nbeg; gend = nend;
          gn = windows(gbeg, gend);
          nr = nnr;
          nbeg = nend = 0;
          if (nr >= 0) { nbeg = __ldg(q.row_offsets + nr); nend = __ldg(q.row_offsets + nr + 1); }
          nnr = row_at(gt + 2);
        }
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int d = 0; d + 1 < kStages; ++d) produce(ring + d * kStage);

    if constexpr (VDN) {
      const bool ok = mbar_wait(bar, phase, &s_abort, q.status, 20);
      if (!__syncthreads_and(ok)) {
        for (int i = 0; i < 1000 && !mbar_try_wait(bar, phase); ++i) __nanosleep(1000);
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        return;
      }
    } else {
      VT* sm = reinterpret_cast<VT*>(slice_smem);
      const VT* src = static_cast<const VT*>(q.dense) + static_cast<size_t>(z) * q.k * q.n + c0;
#pragma unroll 16
      for (int i = threadIdx.x; i < q.k * kWidth; i += kThreads) {
        const int r = i / kWidth, c = i % kWidth;
        sm[i] = c < width ? __ldg(src + static_cast<size_t>(r) * q.n + c) : VT(0);
      }
      __syncthreads();
    }

    VT* out = static_cast<VT*>(q.out) + static_cast<size_t>(z) * q.m * q.n + c0 + sl * CPL;
    constexpr int kAcc = CPL > 1 ? CPL / 2 : 1;
    float2 acc[kAcc];
#pragma unroll
    for (int j = 0; j < kAcc; ++j) acc[j] = make_float2(0.f, 0.f);
    uint32_t stage = ring;
    for (int t = 0; t < rounds;) {
      asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
      __syncwarp();  // this window is here, and the one before it has been read
      produce(stage == ring ? ring + (kStages - 1) * kStage : stage - kStage);
      const uint4 head = lds128(stage + sub * 16u);
      const int r = static_cast<int>(head.x), beg = static_cast<int>(head.y), end = static_cast<int>(head.z);
      const int w = abs(static_cast<int>(head.w)) - 1;
      const bool last = static_cast<int>(head.w) < 0;
      const int base = (beg & ~(VN - 1)) + w * kWin;
      // packs of this window: all of them, and those that are whole in every row
      int packs = min(max((end - base + VN - 1) / VN, 0), kPacks), from = base < beg ? 1 : 0;
      int to = min(max((end - base) / VN, 0), kPacks);
      if constexpr (S > 1) {
        packs = __reduce_max_sync(0xffffffffu, packs);
        from = __reduce_max_sync(0xffffffffu, from);
        to = __reduce_min_sync(0xffffffffu, to);
      }
      const uint32_t vat = stage + S * 16u + sub * kSub, cat = vat + kWin * static_cast<uint32_t>(sizeof(VT));
      auto pack = [&](int i, bool whole) {
        const uint4 rv = lds128(vat + i * 16u);
        uint4 rc[kIdx];
#pragma unroll
        for (int j = 0; j < kIdx; ++j) rc[j] = lds128(cat + (i * kIdx + j) * 16u);
        float v[VN];
        LaneWord<B> x[VN];
#pragma unroll
        for (int e = 0; e < VN; ++e) {
          v[e] = to_float(reinterpret_cast<const VT*>(&rv)[e]);
          uint32_t at = mine + static_cast<uint32_t>(to_index(reinterpret_cast<const IT*>(rc)[e])) * kRow;
          if (!whole) {
            const int p = base + i * VN + e;
            if (p < beg || p >= end) { at = zero_row; v[e] = 0.f; }
          }
          x[e] = lds<B>(at);
        }
#pragma unroll
        for (int e = 0; e < VN; ++e) {
          if constexpr (sizeof(VT) == 4 && B == 4) {
            acc[0].x = fmaf(v[e], __uint_as_float(x[e].x[0]), acc[0].x);
          } else if constexpr (sizeof(VT) == 4) {
#pragma unroll
            for (int j = 0; j < kAcc; ++j)
              acc[j] = ffma2(make_float2(v[e], v[e]),
                             make_float2(__uint_as_float(x[e].x[2 * j]), __uint_as_float(x[e].x[2 * j + 1])), acc[j]);
          } else {
#pragma unroll
            for (int j = 0; j < kAcc; ++j)
              acc[j] = ffma2(make_float2(v[e], v[e]), __half22float2(reinterpret_cast<const __half2&>(x[e].x[j])), acc[j]);
          }
        }
      };
      int i = 0;
      if (from > 0 && packs > 0) { pack(0, false); i = 1; }
#pragma unroll 4
      for (; i < to; ++i) pack(i, true);
      for (; i < packs; ++i) pack(i, false);
      if (last) {
        ++t;
        if (r >= 0 && sl * CPL < width) {
          float res[CPL];
#pragma unroll
          for (int j = 0; j < CPL; ++j) res[j] = j % 2 ? acc[j / 2].y : acc[j / 2].x;
          VT* dst = out + static_cast<size_t>(r) * q.n;
          if (q.bias != nullptr) {
            const float bias_r = __ldg(q.bias + r);
#pragma unroll
            for (int j = 0; j < CPL; ++j) { res[j] += bias_r; res[j] = res[j] > 0.f ? res[j] : 0.f; }
          }
          bool stored = false;
          if constexpr (sizeof(VT) == 4) {
            if (q.accumulate) {
#pragma unroll
              for (int j = 0; j < CPL; ++j)
                if (sl * CPL + j < width) atomicAdd(reinterpret_cast<float*>(dst) + j, res[j]);
              stored = true;
            }
          }
          if (stored) {
          } else if (VDN) {
            LaneWord<B> word;
            if constexpr (sizeof(VT) == 4) {
#pragma unroll
              for (int j = 0; j < CPL; ++j) word.x[j] = __float_as_uint(res[j]);
            } else {
#pragma unroll
              for (int j = 0; j < CPL / 2; ++j) {
                const __half2 h = __floats2half2_rn(res[2 * j], res[2 * j + 1]);
                word.x[j] = reinterpret_cast<const uint32_t&>(h);
              }
            }
            if constexpr (B == 4) *reinterpret_cast<uint32_t*>(dst) = word.x[0];
            if constexpr (B == 8) *reinterpret_cast<uint2*>(dst) = make_uint2(word.x[0], word.x[1]);
            if constexpr (B == 16) *reinterpret_cast<uint4*>(dst) = make_uint4(word.x[0], word.x[1], word.x[2], word.x[3]);
          } else {
#pragma unroll
            for (int j = 0; j < CPL; ++j)
              if (sl * CPL + j < width) {
                if constexpr (sizeof(VT) == 4) dst[j] = res[j]; else dst[j] = __float2half_rn(res[j]);
              }
          }
        }
#pragma unroll
        for (int j = 0; j < kAcc; ++j) acc[j] = make_float2(0.f, 0.f);
      }
      stage = stage == ring + (kStages - 1) * kStage ? ring : stage + kStage;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
  }
}

template <typename VT, typename IT, int W, int B>
int slice_bytes(int k) {  // dynamic shared memory, 0 if the slice does not fit
  const long long rows = (static_cast<long long>(k) + kBoxRows - 1) / kBoxRows * kBoxRows;
  const long long bytes = rows * W + 128 + kWarps * kStages * stage_bytes<VT, IT, W, B>();
  return bytes + 128 <= kSmemBytes ? static_cast<int>(bytes) : 0;
}

struct Plan {
  int width;   // bytes of a slice's row: 128, or 64 or 32 where the matrix is not wider or the slice would not fit; 0: none fits
  int lane;    // bytes of a lane
  int groups;  // CTAs that share an item (slice, batch item), each with some of the rows
  double us;   // the time it should take
};

// Fitted on B200 (fp32 / fp16): a CTA takes 1.0 / 1.55 ns for a nonzero of a 128-byte slice, 0.46 / 0.92 ns for narrower
// ones, and never less than 33 ns for each nonzero of an average row, since the longest is walked by one warp; the slice
// arrives at 115 GB/s (scalar loads: 10 elements a nanosecond); launch and start take 2.3 us.
template <typename VT, typename IT>
Plan make_plan(int m, int k, int n, int nnz, bool vdn, int batch) {
  Plan p{};
  const long long bytes = static_cast<long long>(n) * static_cast<int>(sizeof(VT));
  p.width = bytes > 64 ? 128 : bytes > 32 ? 64 : 32;
  if (p.width == 128 && slice_bytes<VT, IT, 128, 8>(k) == 0) p.width = 64;
  if (p.width == 64 && slice_bytes<VT, IT, 64, 8>(k) == 0) p.width = 32;
  if ((p.width == 32 && slice_bytes<VT, IT, 32, 8>(k) == 0) || m == 0 || n == 0 || nnz == 0 || batch == 0) {
    p.width = 0;
    p.us = 1e30;
    return p;
  }
  const bool f32 = sizeof(VT) == 4;
  const int cols = p.width / static_cast<int>(sizeof(VT));
  const long long items = static_cast<long long>((n + cols - 1) / cols) * batch;
  const double row = static_cast<double>(nnz) / m;
  const double each = p.width == 128 ? (f32 ? 1.0e-3 : 1.55e-3) : (f32 ? 0.46e-3 : 0.92e-3);
  const double fill = 0.3 + k * p.width / 115e3 + (vdn ? 0.0 : 1e-4 * k * cols);
  p.us = 1e30;
  long long rounds = (items + kNumSMs - 1) / kNumSMs;
  for (int i = 0; i < 4; ++i, ++rounds) {
    const int g = static_cast<int>(std::max(1ll, std::min<long long>(rounds * kNumSMs / items, (m + 1) / 2)));
    const double t = rounds * (fill + std::max(each * nnz / g + (f32 ? 0.02 : 0.012) * row, 0.033 * row));
    if (t < p.us) { p.us = t; p.groups = g; }
  }
  p.us += 2.0;
  // Eight bytes a lane cost less for a nonzero (the values and columns are read for more rows at a time), but make
  // bunches of twice the rows, which want to be enough for every warp.
  p.lane = m / (32 * 8 / p.width) >= p.groups * kWarps ? 8 : 4;
  return p;
}

template <typename VT, typename IT, int W, int B, bool VDN>
int launch(Params q, int batch, cudaStream_t stream) {
  auto kern = spmm_slice_kernel<VT, IT, W, B, VDN>;
  constexpr int kWidth = W / static_cast<int>(sizeof(VT));
  {
    static std::mutex mutex;
    static bool configured[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) dev = -1;
    std::lock_guard<std::mutex> lock(mutex);
    if (dev < 0 || dev >= 64 || !configured[dev]) {
      const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes - 128);
      if (e != cudaSuccess) return static_cast<int>(e);
      if (dev >= 0 && dev < 64) configured[dev] = true;
    }
  }
  CUtensorMap map{};
  if (VDN) {
    const int st = make_map_slice(&map, sizeof(VT) == 2, q.dense, static_cast<long long>(batch) * q.k, q.n, kBoxRows, kWidth);
    if (st != IEX_OK) return st;
  }
  q.status = status_word();
  if (!q.status) return IEX_ERR_DRIVER;
  q.tiles = (q.n + kWidth - 1) / kWidth;
  const long long units = static_cast<long long>(q.tiles) * batch * q.groups;
  if (units > 0x7fffffffll - kNumSMs) return IEX_ERR_UNSUPPORTED;
  q.units = static_cast<int>(units);
  return launch_overlapped(kern, dim3(std::min(q.units, kNumSMs)), dim3(kWarps * 32), slice_bytes<VT, IT, W, B>(q.k), stream,
                           map, q);
}

template <typename VT, typename IT, int W>
int launch_width(const Params& q, int lane, bool vdn, int batch, cudaStream_t stream) {
  if (lane == 8) return vdn ? launch<VT, IT, W, 8, true>(q, batch, stream) : launch<VT, IT, W, 8, false>(q, batch, stream);
  return vdn ? launch<VT, IT, W, 4, true>(q, batch, stream) : launch<VT, IT, W, 4, false>(q, batch, stream);
}

}  // namespace

// The time spmm_slice should take, us; 1e30 where no slice fits.
template <typename VT, typename IT>
double spmm_slice_us(int m, int k, int n, int nnz, bool vdn, int batch) {
  return make_plan<VT, IT>(m, k, n, nnz, vdn, batch).us;
}

template <typename VT, typename IT>
int spmm_slice(int m, int k, int n, int nnz, const int* row_indices, const VT* values, long long vstride,
               const int* row_offsets, const IT* cols, const VT* dense, const float* bias, VT* out, int batch,
               int accumulate, cudaStream_t stream) {
  Params q{};
  q.m = m; q.k = k; q.n = n; q.nnz = nnz;
  q.row_indices = row_indices;
  q.values = values; q.values_batch_stride = vstride; q.row_offsets = row_offsets; q.cols = cols;
  q.dense = dense; q.bias = bias; q.out = out; q.accumulate = accumulate;
  const bool vdn = n % (16 / sizeof(VT)) == 0 && aligned16(dense) && aligned16(out);
  const Plan p = make_plan<VT, IT>(m, k, n, nnz, vdn, batch);
  q.groups = p.groups;
  switch (p.width) {
    case 128: return launch_width<VT, IT, 128>(q, p.lane, vdn, batch, stream);
    case 64: return launch_width<VT, IT, 64>(q, p.lane, vdn, batch, stream);
    case 32: return launch_width<VT, IT, 32>(q, p.lane, vdn, batch, stream);
  }
  return IEX_ERR_UNSUPPORTED;
}

template int spmm_slice<float, int>(int, int, int, int, const int*, const float*, long long, const int*, const int*, const float*,
                                    const float*, float*, int, int, cudaStream_t);
template int spmm_slice<__half, int>(int, int, int, int, const int*, const __half*, long long, const int*, const int*, const __half*,
                                     const float*, __half*, int, int, cudaStream_t);
template int spmm_slice<__half, uint16_t>(int, int, int, int, const int*, const __half*, long long, const int*, const uint16_t*,
                                          const __half*, const float*, __half*, int, int, cudaStream_t);

template double spmm_slice_us<float, int>(int, int, int, int, bool, int);
template double spmm_slice_us<__half, int>(int, int, int, int, bool, int);
template double spmm_slice_us<__half, uint16_t>(int, int, int, int, bool, int);

}  // namespace iex
