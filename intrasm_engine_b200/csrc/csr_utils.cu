// CSR <-> dense helpers on the device.
//   * csr_to_dense (fp16): where an activation CSR becomes the tile operand of the
//     tensor-core linear (ReLU-sparse FFN down projection).
//   * dense_to_csr (fp16 / fp32, optional ReLU): builds row_offsets, the row visiting order
//     (rows by decreasing nnz, ties in row order), values and ascending column indices of a
//     dense matrix in two calls: "count" (row lengths, offsets, row order) and, once the
//     caller has read nnz = row_offsets[m] and allocated the arrays, "fill".
#include "common.cuh"

namespace iex {
namespace {

__device__ __forceinline__ bool keeps(float v, bool relu) { return relu ? v > 0.f : v != 0.f; }

// One warp per row: number of stored elements of the row.
template <typename T>
__global__ void __launch_bounds__(256)
row_count_kernel(int m, int k, const T* __restrict__ dense, int relu, int* __restrict__ row_nnz) {
  const int lane = threadIdx.x & 31;
  const int warps = (gridDim.x * blockDim.x) >> 5;
  for (int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < m; r += warps) {
    const T* row = dense + static_cast<size_t>(r) * k;
    int cnt = 0;
    for (int c0 = 0; c0 < k; c0 += 32) {
      const int c = c0 + lane;
      const bool on = c < k && keeps(to_float(row[c]), relu != 0);
      cnt += __popc(__ballot_sync(0xffffffffu, on));
    }
    if (lane == 0) row_nnz[r] = cnt;
  }
}

// One block: row_offsets[0..m] = exclusive prefix sum of row_nnz (chunks of 1024 rows).
__global__ void __launch_bounds__(1024) row_scan_kernel(int m, const int* __restrict__ row_nnz,
                                                        int* __restrict__ row_offsets) {
  __shared__ int warp_sums[32];
  __shared__ int carry_s;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) { carry_s = 0; row_offsets[0] = 0; }
  __syncthreads();
  for (int base = 0; base < m; base += 1024) {
    const int i = base + threadIdx.x;
    const int v = i < m ? row_nnz[i] : 0;
    int x = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, d);
      if (lane >= d) x += y;
    }
    if (lane == 31) warp_sums[warp] = x;
    __syncthreads();
    if (warp == 0) {
      int w = warp_sums[lane];
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, w, d);
        if (lane >= d) w += y;
      }
      warp_sums[lane] = w;
    }
    __syncthreads();
    const int incl = x + (warp > 0 ? warp_sums[warp - 1] : 0) + carry_s;
    if (i < m) row_offsets[i + 1] = incl;
    __syncthreads();
    if (threadIdx.x == 1023) carry_s = incl;
    __syncthreads();
  }
}

// Row visiting order: position of row r = number of rows with more nonzeros, plus the rows
// before r with as many (a stable descending sort, computed as a rank: every thread compares
// its row with all others, staged through shared memory in chunks).
__global__ void __launch_bounds__(256) row_rank_kernel(int m, const int* __restrict__ row_nnz,
                                                       int* __restrict__ row_indices) {
  __shared__ int chunk[1024];
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  const int mine = r < m ? row_nnz[r] : 0;
  int rank = 0;
  for (int base = 0; base < m; base += 1024) {
    for (int i = threadIdx.x; i < 1024; i += blockDim.x) chunk[i] = base + i < m ? row_nnz[base + i] : -1;
    __syncthreads();
    const int lim = min(1024, m - base);
    for (int i = 0; i < lim; ++i) {
      const int o = chunk[i];
      rank += (o > mine || (o == mine && base + i < r)) ? 1 : 0;
    }
    __syncthreads();
  }
  if (r < m) row_indices[rank] = r;
}

// One warp per row: stored elements and their column indices, in column order.
template <typename T, typename IT>
__global__ void __launch_bounds__(256)
row_fill_kernel(int m, int k, const T* __restrict__ dense, int relu, const int* __restrict__ row_offsets,
                T* __restrict__ values, IT* __restrict__ cols) {
  const int lane = threadIdx.x & 31;
  const int warps = (gridDim.x * blockDim.x) >> 5;
  for (int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < m; r += warps) {
    const T* row = dense + static_cast<size_t>(r) * k;
    int pos = row_offsets[r];
    for (int c0 = 0; c0 < k; c0 += 32) {
      const int c = c0 + lane;
      const T v = c < k ? row[c] : T(0);
      const bool on = c < k && keeps(to_float(v), relu != 0);
      const unsigned b = __ballot_sync(0xffffffffu, on);
      if (on) {
        const int p = pos + __popc(b & ((1u << lane) - 1u));
        values[p] = v;
        cols[p] = static_cast<IT>(c);
      }
      pos += __popc(b);
    }
  }
}

// CTA (x, y) owns the columns [y * slice, (y + 1) * slice) of rows x, x + gridDim.x, ...: it
// clears its piece of the dense row with 128-bit stores and then writes the row's nonzeros
// that fall into it.  A few CTAs per row instead of one keep each CTA's work down to one or
// two instructions per thread, so the kernel is as long as its chain of three dependent memory
// round trips (row offsets, indices and values, stores) and no longer; the row's offsets and
// its first indices and values are requested before the clearing stores, not after.
template <typename IT>
__global__ void __launch_bounds__(256)
csr_to_dense_f16_kernel(int m, int k, int slice, const int* __restrict__ row_offsets, const IT* __restrict__ cols,
                        const __half* __restrict__ values, __half* __restrict__ out, int mark) {
  grid_dependency_wait();  // `out` may still be read by the kernel before this one
  grid_launch_dependents();
  const int c0 = blockIdx.y * slice;
  const int c1 = c0 + slice < k ? c0 + slice : k;
  const bool vec = (k & 7) == 0 && (slice & 7) == 0 && (reinterpret_cast<uintptr_t>(out) & 15u) == 0;
  for (int r = blockIdx.x; r < m; r += gridDim.x) {
    __half* row = out + static_cast<size_t>(r) * k;
    const int beg = __ldg(row_offsets + r), end = __ldg(row_offsets + r + 1);
    int p = beg + threadIdx.x;
    int c = -1;
    __half v = __float2half(0.f);
    if (p < end) {
      c = to_index(__ldg(cols + p));
      v = __ldg(values + p);
    }
    if (vec) {
      uint4* row4 = reinterpret_cast<uint4*>(row);
      for (int i = (c0 >> 3) + threadIdx.x; i < (c1 >> 3); i += blockDim.x) row4[i] = make_uint4(0u, 0u, 0u, 0u);
    } else {
      for (int i = c0 + threadIdx.x; i < c1; i += blockDim.x) row[i] = __float2half(0.f);
    }
    __syncthreads();
    bool unordered = false;
    while (p < end) {
      if (c >= c0 && c < c1) row[c] = v;
      if (mark && p > beg && to_index(__ldg(cols + p - 1)) >= c) unordered = true;
      p += blockDim.x;
      if (p < end) {
        c = to_index(__ldg(cols + p));
        v = __ldg(values + p);
      }
    }
    if (!mark) {
      __syncthreads();
    } else if (__syncthreads_or(unordered ? 1 : 0)) {
      // a column may be there twice: all that the row stores is marked, and summed from the positions
      for (p = beg + threadIdx.x; p < end; p += blockDim.x) {
        c = to_index(__ldg(cols + p));
        if (c >= c0 && c < c1) row[c] = __ushort_as_half(0x7fff);
      }
      __syncthreads();
    }
  }
}

// The same for matrices of many rows: TPR threads (a warp, or a block where a row needs more shared memory)
// build a row in shared memory and store it with 16-byte pieces, so the dense row is written once
// instead of cleared and then scattered into.  Neighbouring lanes take neighbouring pairs of nonzeros:
// the pair loads are coalesced, and because columns ascend the two-byte shared-memory stores of a warp
// fall into neighbouring banks.  kU pairs per thread are requested before the first store; a first or last
// nonzero whose partner belongs to another row is written alone, so the loop has no checks.
// 11008 x 4096 at 50 %, 180 MB: 63 us as a block per row with a check per pair.
template <typename IT>
__device__ __forceinline__ void load_pair(const __half* values, const IT* cols, int p, uint32_t& v, int (&c)[2]) {
  v = __ldg(reinterpret_cast<const uint32_t*>(values + p));
  if constexpr (sizeof(IT) == 2) {
    const uint32_t cc = __ldg(reinterpret_cast<const uint32_t*>(cols + p));
    c[0] = static_cast<int>(cc & 0xffffu);
    c[1] = static_cast<int>(cc >> 16);
  } else {
    const int2 cc = __ldg(reinterpret_cast<const int2*>(cols + p));
    c[0] = cc.x;
    c[1] = cc.y;
  }
}

// A row that is not strictly ascending, built again (all TPR threads): NaN where a column is stored twice.  Two bits per
// column first (seen, seen again), then the marks, then the values of the other columns.
template <typename IT, int TPR, typename Sync>
__device__ __noinline__ void mark_repeats(uint32_t* words, int ld, int beg, int end, int t, const IT* cols, const __half* values,
                                          const Sync& sync) {
  for (int i = t; i < ld / 2; i += TPR) words[i] = 0u;
  sync();
  for (int p = beg + t; p < end; p += TPR) {
    const int c = to_index(__ldg(cols + p)), at = 16 * (c & 1);
    if (atomicOr(words + (c >> 1), 1u << at) >> at & 1u) atomicOr(words + (c >> 1), 2u << at);
  }
  sync();
  for (int i = t; i < ld / 2; i += TPR) words[i] = (words[i] & 2u ? 0x7fffu : 0u) | (words[i] & 0x20000u ? 0x7fff0000u : 0u);
  sync();
  unsigned short* row = reinterpret_cast<unsigned short*>(words);
  for (int p = beg + t; p < end; p += TPR) {
    const int c = to_index(__ldg(cols + p));
    if (row[c] != 0x7fffu) row[c] = __half_as_ushort(__ldg(values + p));
  }
  sync();
}

// kMark: the copy is for a product that sums NaN outputs again from the stored positions (csr_terms.cuh).  A column that a row
// stores twice, of which only one value would be in the copy, becomes NaN, so that its outputs are.
template <typename IT, int TPR, bool kMark>
__global__ void __launch_bounds__(256)
csr_expand_rows_kernel(int m, int ld, const int* __restrict__ row_offsets, const IT* __restrict__ cols,
                       const __half* __restrict__ values, __half* __restrict__ out) {
  constexpr int kU = TPR == 32 ? 8 : 4;
  extern __shared__ __align__(16) uint8_t row_smem[];
  const int group = threadIdx.x / TPR, t = threadIdx.x % TPR;
  const int groups = blockDim.x / TPR;
  uint8_t* buf = row_smem + group * (static_cast<uint32_t>(ld) * 2u);
  __half* row_buf = reinterpret_cast<__half*>(buf);
  uint4* row_vec = reinterpret_cast<uint4*>(buf);
  const int vecs = ld >> 3;
  auto sync = [] { if constexpr (TPR == 32) __syncwarp(); else __syncthreads(); };
  auto put = [&](uint32_t v, const int (&c)[2]) {
    row_buf[c[0]] = __ushort_as_half(static_cast<unsigned short>(v & 0xffffu));
    row_buf[c[1]] = __ushort_as_half(static_cast<unsigned short>(v >> 16));
  };
  for (int i = t; i < vecs; i += TPR) row_vec[i] = make_uint4(0u, 0u, 0u, 0u);
  grid_dependency_wait();
  grid_launch_dependents();
  sync();
  const int step = gridDim.x * groups;
  int r = blockIdx.x * groups + group;
  int beg = 0, end = 0;
  if (r < m) { beg = __ldg(row_offsets + r); end = __ldg(row_offsets + r + 1); }
  for (; r < m; r += step) {
    int next_beg = 0, next_end = 0;
    if (r + step < m) { next_beg = __ldg(row_offsets + r + step); next_end = __ldg(row_offsets + r + step + 1); }
    const int even_beg = (beg + 1) & ~1, even_end = end & ~1;
    // A pair against itself and the position before it, which the lane before has; lane 0 has it from the window before, or,
    // where another warp has that, loads it.  Called by whole warps.
    bool unordered = false;
    int before = kMark && (beg & 1) && beg < end ? to_index(__ldg(cols + beg)) : -1;
    auto check = [&](int p, bool on, const int (&c)[2]) {
      if constexpr (kMark) {
        const int lane = threadIdx.x & 31;
        const int rotated = __shfl_sync(0xffffffffu, c[1], (lane + 31) & 31);
        int prev = rotated;
        if (lane == 0) prev = TPR == 32 || p == even_beg ? before : on ? to_index(__ldg(cols + p - 1)) : -1;
        unordered = unordered || (on && (prev >= c[0] || c[0] >= c[1]));
        if (TPR == 32) before = rotated;
      }
    };
    if (kMark && t == 1 && (end & 1) && end - 1 > beg) unordered = to_index(__ldg(cols + end - 2)) >= to_index(__ldg(cols + end - 1));
    if (t == 0 && beg < end && (beg & 1)) row_buf[to_index(__ldg(cols + beg))] = __ldg(values + beg);
    if (t == 1 && beg < end && (end & 1) && end - 1 >= even_beg) row_buf[to_index(__ldg(cols + end - 1))] = __ldg(values + end - 1);
    int p0 = even_beg;
    for (; p0 + 2 * TPR * kU <= even_end; p0 += 2 * TPR * kU) {
      uint32_t v[kU];
      int c[kU][2];
#pragma unroll
      for (int u = 0; u < kU; ++u) load_pair(values, cols, p0 + 2 * TPR * u + 2 * t, v[u], c[u]);
#pragma unroll
      for (int u = 0; u < kU; ++u) {
        put(v[u], c[u]);
        check(p0 + 2 * TPR * u + 2 * t, true, c[u]);
      }
    }
    if (p0 < even_end) {
      uint32_t v[kU];
      int c[kU][2] = {};
#pragma unroll
      for (int u = 0; u < kU; ++u)
        if (p0 + 2 * TPR * u + 2 * t < even_end) load_pair(values, cols, p0 + 2 * TPR * u + 2 * t, v[u], c[u]);
#pragma unroll
      for (int u = 0; u < kU; ++u)
      {
        const int p = p0 + 2 * TPR * u + 2 * t;
        if (p < even_end) put(v[u], c[u]);
        check(p, p < even_end, c[u]);
      }
    }
    if constexpr (kMark) {
      bool again;
      if constexpr (TPR == 32) again = __any_sync(0xffffffffu, unordered);
      else again = __syncthreads_or(unordered ? 1 : 0) != 0;
      if (again) mark_repeats<IT, TPR>(reinterpret_cast<uint32_t*>(buf), ld, beg, end, t, cols, values, sync);
    }
    sync();
    uint4* dst = reinterpret_cast<uint4*>(out + static_cast<size_t>(r) * ld);
#pragma unroll 4
    for (int i = t; i < vecs; i += TPR) {
      dst[i] = row_vec[i];
      row_vec[i] = make_uint4(0u, 0u, 0u, 0u);
    }
    sync();
    beg = next_beg;
    end = next_end;
  }
}

// out[p] = dense[row of p, cols[p]] for every stored position: a warp per row, so that the positions
// of a warp fall into one dense row (columns ascend: neighbouring lanes, neighbouring sectors).
template <typename IT>
__global__ void __launch_bounds__(256)
csr_sample_kernel(int m, long long ld, const int* __restrict__ row_offsets, const IT* __restrict__ cols,
                  const __half* __restrict__ dense, __half* __restrict__ out) {
  const int lane = threadIdx.x & 31;
  grid_dependency_wait();
  grid_launch_dependents();
  for (int r = blockIdx.x * 8 + (threadIdx.x >> 5); r < m; r += gridDim.x * 8) {
    const int beg = __ldg(row_offsets + r), end = __ldg(row_offsets + r + 1);
    const __half* row = dense + static_cast<size_t>(r) * ld;
    for (int p0 = beg; p0 < end; p0 += 128) {
      int c[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int p = p0 + 32 * u + lane;
        c[u] = p < end ? to_index(__ldg(cols + p)) : 0;
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int p = p0 + 32 * u + lane;
        if (p < end) out[p] = __ldg(row + c[u]);
      }
    }
  }
}

// out[i] = in[perm[i]]: the values of a pattern in the order of its transpose.  Bound by the sectors of `in` that the
// gathers touch; four per thread in flight.  234 k fp32 values: 4.6 -> 2.4 us, and 5 us less of host time than the
// library's indexing.
template <typename T>
__global__ void __launch_bounds__(256)
gather_values_kernel(int count, const T* __restrict__ in, const long long* __restrict__ perm, T* __restrict__ out) {
  grid_dependency_wait();
  grid_launch_dependents();
  const long long base = blockIdx.x * 1024ll + threadIdx.x;
  long long at[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) at[u] = base + 256 * u < count ? __ldg(perm + base + 256 * u) : 0;
  T v[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) v[u] = __ldg(in + at[u]);
#pragma unroll
  for (int u = 0; u < 4; ++u)
    if (base + 256 * u < count) out[base + 256 * u] = v[u];
}

// Rows of `cols` fp16 values, any alignment, into rows of `ld` (a multiple of 8), the rest zero.
__global__ void __launch_bounds__(256)
pad_rows_kernel(int rows, int cols, int ld, const __half* __restrict__ in, __half* __restrict__ out) {
  grid_dependency_wait();
  grid_launch_dependents();
  const int vecs = ld >> 3;
  for (long long i = blockIdx.x * 256ll + threadIdx.x; i < static_cast<long long>(rows) * vecs; i += gridDim.x * 256ll) {
    const long long r = i / vecs;
    const int c = static_cast<int>(i - r * vecs) * 8;
    const __half* src = in + r * cols + c;
    uint4 pk;
    __half* h = reinterpret_cast<__half*>(&pk);
#pragma unroll
    for (int e = 0; e < 8; ++e) h[e] = c + e < cols ? __ldg(src + e) : __float2half(0.f);
    reinterpret_cast<uint4*>(out)[i] = pk;
  }
}

// max(x, 0) on 16-byte pieces (NaN and negative values become 0, as in the ReLU of the converter).  An input that is only
// aligned to its elements (a view into a larger buffer) is read value by value.
template <bool kVec>
__global__ void __launch_bounds__(256)
relu_f16_kernel(long long vecs, const __half* __restrict__ in, uint4* __restrict__ out) {
  grid_dependency_wait();
  grid_launch_dependents();
  const __half zero = __float2half(0.f);
  for (long long i = blockIdx.x * 256ll + threadIdx.x; i < vecs; i += gridDim.x * 256ll) {
    uint4 v;
    __half* h = reinterpret_cast<__half*>(&v);
    if constexpr (kVec) {
      v = __ldg(reinterpret_cast<const uint4*>(in) + i);
    } else {
#pragma unroll
      for (int e = 0; e < 8; ++e) h[e] = __ldg(in + 8 * i + e);
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) h[e] = __hgt(h[e], zero) ? h[e] : zero;
    out[i] = v;
  }
}

// CSR sanity check.  Threads stride over rows (offset rules, row order entries) and over
// nonzeros (column range, ascending order inside a row: position p belongs to a row boundary
// exactly when some offset equals p, which a binary search over row_offsets answers).
// Violations are OR-ed into one device word.
template <typename IT>
__global__ void __launch_bounds__(256)
csr_validate_kernel(int m, int k, int nnz, const int* __restrict__ row_offsets, const IT* __restrict__ cols,
                    const int* __restrict__ row_indices, int require_ascending, int* __restrict__ result) {
  const int tid = blockIdx.x * blockDim.x + threadIdx.x;
  const int nthreads = gridDim.x * blockDim.x;
  int bad = 0;
  if (tid == 0) {
    if (row_offsets[0] != 0) bad |= IEX_CSR_BAD_FIRST_OFFSET;
    if (row_offsets[m] != nnz) bad |= IEX_CSR_BAD_LAST_OFFSET;
  }
  for (int r = tid; r < m; r += nthreads) {
    const int a = row_offsets[r], b = row_offsets[r + 1];
    if (b < a || a < 0 || b > nnz) bad |= IEX_CSR_OFFSETS_NOT_MONOTONE;
    if (row_indices != nullptr) {
      const int v = row_indices[r];
      if (v < 0 || v >= m) bad |= IEX_CSR_BAD_ROW_INDEX;
    }
  }
  for (int p = tid; p < nnz; p += nthreads) {
    const int c = to_index(cols[p]);
    if (c < 0 || c >= k) bad |= IEX_CSR_COLUMN_OUT_OF_RANGE;
    if (require_ascending && p > 0) {
      // is p the first nonzero of a row?  largest r with row_offsets[r] <= p ...
      int lo = 0, hi = m;
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (row_offsets[mid] <= p) lo = mid; else hi = mid - 1;
      }
      // ... starts the row holding p; p continues a row when that offset is below p
      if (row_offsets[lo] < p && to_index(cols[p - 1]) >= c) bad |= IEX_CSR_COLUMNS_NOT_ASCENDING;
    }
  }
  if (bad) atomicOr(result, bad);
}

}  // namespace
}  // namespace iex

extern "C" int iex_csr_validate(int m, int k, int nnz, const int32_t* row_offsets, const void* column_indices,
                                int index_bits, const int32_t* row_indices, int require_ascending,
                                int32_t* result, void* stream) {
  using namespace iex;
  if (m < 0 || k < 0 || nnz < 0 || (index_bits != 16 && index_bits != 32)) return IEX_ERR_BAD_ARG;
  if (!row_offsets || !result || (nnz > 0 && !column_indices)) return IEX_ERR_BAD_ARG;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  cudaError_t e = cudaMemsetAsync(result, 0, sizeof(int32_t), s);
  if (e != cudaSuccess) return static_cast<int>(e);
  const long long work = static_cast<long long>(nnz) > m ? nnz : m;
  long long blocks = (work + 255) / 256;
  blocks = blocks < 1 ? 1 : (blocks > 8 * kNumSMs ? 8 * kNumSMs : blocks);
  if (index_bits == 16)
    csr_validate_kernel<uint16_t><<<static_cast<int>(blocks), 256, 0, s>>>(
        m, k, nnz, row_offsets, static_cast<const uint16_t*>(column_indices), row_indices, require_ascending,
        result);
  else
    csr_validate_kernel<int><<<static_cast<int>(blocks), 256, 0, s>>>(
        m, k, nnz, row_offsets, static_cast<const int*>(column_indices), row_indices, require_ascending, result);
  return launch_status();
}

namespace iex {
namespace {

template <typename IT>
int csr_to_dense(int m, int ld, const int* row_offsets, const IT* cols, const __half* values, __half* out, bool mark,
                 cudaStream_t s) {
  // Many rows, or short ones: one pass through shared memory.  A few long rows: column slices, since a block that clears
  // and stores a long row alone takes longer than the second pass (256 x 11008 before a product: 30.6 us in slices, 31.3
  // us by rows; 128 x 6000: 20.4 and 18.3 us).
  const bool pairs = (reinterpret_cast<uintptr_t>(values) & 3u) == 0 &&
                     (reinterpret_cast<uintptr_t>(cols) & (2 * sizeof(IT) - 1)) == 0;
  if (ld % 8 == 0 && ld <= (m >= 4 * kNumSMs ? 24 * 1024 : 6144) && pairs && aligned16(out)) {
    // a warp per row while the rows of 24 warps fit into an SM's shared memory, else a block per row
    if (ld <= 4608 && m >= 4 * kNumSMs) {
      const int row_bytes = 2 * ld, fit = 48 * 1024 / row_bytes;  // a block's default shared memory
      const int warps = fit < 8 ? fit : 8;
      const int per_sm = 220 * 1024 / (row_bytes * warps) < 8 ? 220 * 1024 / (row_bytes * warps) : 8;
      const int blocks = (m + warps - 1) / warps, most = kNumSMs * per_sm;
      return launch_overlapped(mark ? csr_expand_rows_kernel<IT, 32, true> : csr_expand_rows_kernel<IT, 32, false>, dim3(blocks < most ? blocks : most), dim3(32 * warps),
                               static_cast<size_t>(ld) * 2 * warps, s, m, ld, row_offsets, cols, values, out);
    }
    return launch_overlapped(mark ? csr_expand_rows_kernel<IT, 256, true> : csr_expand_rows_kernel<IT, 256, false>, dim3(m < 8 * kNumSMs ? m : 8 * kNumSMs), dim3(256),
                             static_cast<size_t>(ld) * 2, s, m, ld, row_offsets, cols, values, out);
  }
  // about eight CTAs of 256 threads per SM in all: rows first, then up to eight column slices
  // (multiples of 8 columns) per row
  const int gx = m < 8 * kNumSMs ? m : 8 * kNumSMs;
  int slices = (8 * kNumSMs) / gx;
  slices = slices < 1 ? 1 : (slices > 8 ? 8 : slices);
  int slice = ((ld + slices - 1) / slices + 7) & ~7;
  if (slice < 256) slice = 256 < ld ? 256 : ((ld + 7) & ~7);
  return launch_overlapped(csr_to_dense_f16_kernel<IT>, dim3(gx, (ld + slice - 1) / slice), dim3(256), 0, s, m, ld,
                           slice, row_offsets, cols, values, out, mark ? 1 : 0);
}

}  // namespace
}  // namespace iex

static int csr_to_dense_any(int m, int k, int ld, const int32_t* row_offsets, const void* column_indices, int index_bits,
                            const void* values, void* out, bool mark, void* stream) {
  using namespace iex;
  if (m < 0 || k < 0 || ld < k || (index_bits != 16 && index_bits != 32)) return IEX_ERR_BAD_ARG;
  if (m == 0 || k == 0) return IEX_OK;
  if (!row_offsets || !out) return IEX_ERR_BAD_ARG;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const __half* v = static_cast<const __half*>(values);
  __half* o = static_cast<__half*>(out);
  if (index_bits == 16)
    return csr_to_dense<uint16_t>(m, ld, row_offsets, static_cast<const uint16_t*>(column_indices), v, o, mark, s);
  return csr_to_dense<int>(m, ld, row_offsets, static_cast<const int*>(column_indices), v, o, mark, s);
}

extern "C" int iex_csr_to_dense_f16_ld(int m, int k, int ld, const int32_t* row_offsets, const void* column_indices,
                                       int index_bits, const void* values, void* out, void* stream) {
  return csr_to_dense_any(m, k, ld, row_offsets, column_indices, index_bits, values, out, false, stream);
}

extern "C" int iex_csr_expand_f16(int m, int k, int ld, const int32_t* row_offsets, const void* column_indices,
                                  int index_bits, const void* values, void* out, void* stream) {
  return csr_to_dense_any(m, k, ld, row_offsets, column_indices, index_bits, values, out, true, stream);
}

extern "C" int iex_csr_to_dense_f16(int m, int k, const int32_t* row_offsets, const void* column_indices,
                                    int index_bits, const void* values, void* out, void* stream) {
  return iex_csr_to_dense_f16_ld(m, k, k, row_offsets, column_indices, index_bits, values, out, stream);
}

extern "C" int iex_csr_sample_f16(int m, int k, long long ld, const int32_t* row_offsets, const void* column_indices,
                                  int index_bits, const void* dense, void* out, void* stream) {
  using namespace iex;
  if (m < 0 || k < 0 || ld < k || (index_bits != 16 && index_bits != 32)) return IEX_ERR_BAD_ARG;
  if (m == 0) return IEX_OK;
  if (!row_offsets) return IEX_ERR_BAD_ARG;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int grid = (m + 7) / 8 < 8 * kNumSMs ? (m + 7) / 8 : 8 * kNumSMs;
  const __half* d = static_cast<const __half*>(dense);
  if (index_bits == 16)
    return launch_overlapped(csr_sample_kernel<uint16_t>, dim3(grid), dim3(256), 0, s, m, ld, row_offsets,
                             static_cast<const uint16_t*>(column_indices), d, static_cast<__half*>(out));
  return launch_overlapped(csr_sample_kernel<int>, dim3(grid), dim3(256), 0, s, m, ld, row_offsets,
                           static_cast<const int*>(column_indices), d, static_cast<__half*>(out));
}

extern "C" int iex_gather_values(int count, int elt_bytes, const void* in, const long long* perm, void* out, void* stream) {
  using namespace iex;
  if (count < 0 || (elt_bytes != 2 && elt_bytes != 4)) return IEX_ERR_BAD_ARG;
  if (count == 0) return IEX_OK;
  if (!in || !perm || !out) return IEX_ERR_BAD_ARG;
  const dim3 grid((static_cast<unsigned>(count) + 1023u) / 1024u);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (elt_bytes == 4)
    return launch_overlapped(gather_values_kernel<uint32_t>, grid, dim3(256), 0, s, count,
                             static_cast<const uint32_t*>(in), perm, static_cast<uint32_t*>(out));
  return launch_overlapped(gather_values_kernel<uint16_t>, grid, dim3(256), 0, s, count, static_cast<const uint16_t*>(in),
                           perm, static_cast<uint16_t*>(out));
}

extern "C" int iex_pad_rows_f16(int rows, int cols, int ld, const void* in, void* out, void* stream) {
  using namespace iex;
  if (rows < 0 || cols < 0 || ld < cols || ld % 8 != 0) return IEX_ERR_BAD_ARG;
  if (rows == 0 || ld == 0) return IEX_OK;
  if (!in || !out || !aligned16(out)) return IEX_ERR_BAD_ARG;
  const long long blocks = (static_cast<long long>(rows) * (ld / 8) + 255) / 256;
  return launch_overlapped(pad_rows_kernel, dim3(static_cast<unsigned>(blocks < 8 * kNumSMs ? blocks : 8 * kNumSMs)),
                           dim3(256), 0, static_cast<cudaStream_t>(stream), rows, cols, ld,
                           static_cast<const __half*>(in), static_cast<__half*>(out));
}

extern "C" int iex_relu_f16(long long count, const void* in, void* out, void* stream) {
  using namespace iex;
  if (count < 0 || count % 8 != 0) return IEX_ERR_BAD_ARG;
  if (count == 0) return IEX_OK;
  if (!in || !out || !aligned16(out)) return IEX_ERR_BAD_ARG;
  const long long blocks = (count / 8 + 255) / 256;
  return launch_overlapped(aligned16(in) ? relu_f16_kernel<true> : relu_f16_kernel<false>,
                           dim3(static_cast<unsigned>(blocks < 8 * kNumSMs ? blocks : 8 * kNumSMs)), dim3(256), 0,
                           static_cast<cudaStream_t>(stream), count / 8, static_cast<const __half*>(in),
                           static_cast<uint4*>(out));
}

extern "C" int iex_dense_to_csr_count(int m, int k, const void* dense, int value_bits, int relu,
                                      int32_t* row_offsets, int32_t* row_indices, void* stream) {
  using namespace iex;
  if (m < 0 || k < 0 || (value_bits != 16 && value_bits != 32)) return IEX_ERR_BAD_ARG;
  if (!row_offsets || !row_indices || (m > 0 && k > 0 && !dense)) return IEX_ERR_BAD_ARG;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  // the row lengths go to row_offsets[1..m], are ranked from there, then scanned in place
  int* lengths = row_offsets + 1;
  if (m > 0) {
    const int blocks = (m + 7) / 8 < 8 * kNumSMs ? (m + 7) / 8 : 8 * kNumSMs;
    if (value_bits == 16)
      row_count_kernel<__half><<<blocks, 256, 0, s>>>(m, k, static_cast<const __half*>(dense), relu, lengths);
    else
      row_count_kernel<float><<<blocks, 256, 0, s>>>(m, k, static_cast<const float*>(dense), relu, lengths);
    int st = launch_status();
    if (st) return st;
    row_rank_kernel<<<(m + 255) / 256, 256, 0, s>>>(m, lengths, row_indices);
    st = launch_status();
    if (st) return st;
  }
  row_scan_kernel<<<1, 1024, 0, s>>>(m, lengths, row_offsets);  // in place: reads [i+1], writes [i+1]
  return launch_status();
}

extern "C" int iex_dense_to_csr_fill(int m, int k, const void* dense, int value_bits, int relu,
                                     const int32_t* row_offsets, void* values, void* column_indices,
                                     int index_bits, void* stream) {
  using namespace iex;
  if (m < 0 || k < 0 || (value_bits != 16 && value_bits != 32) || (index_bits != 16 && index_bits != 32))
    return IEX_ERR_BAD_ARG;
  if (index_bits == 16 && k > 65536) return IEX_ERR_UNSUPPORTED;
  if (m == 0 || k == 0) return IEX_OK;
  if (!dense || !row_offsets || !values || !column_indices) return IEX_ERR_BAD_ARG;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int blocks = (m + 7) / 8 < 8 * kNumSMs ? (m + 7) / 8 : 8 * kNumSMs;
#define IEX_FILL(T, IT)                                                                              \
  row_fill_kernel<T, IT><<<blocks, 256, 0, s>>>(m, k, static_cast<const T*>(dense), relu, row_offsets, \
                                                static_cast<T*>(values), static_cast<IT*>(column_indices))
  if (value_bits == 16 && index_bits == 16) IEX_FILL(__half, uint16_t);
  else if (value_bits == 16) IEX_FILL(__half, int);
  else if (index_bits == 16) IEX_FILL(float, uint16_t);
  else IEX_FILL(float, int);
#undef IEX_FILL
  return launch_status();
}
