// Dense fp16 linear layer for a handful of tokens: out[t, o] = sum_c x[t, c] * w[o, c], fp32 accumulation.
//
// A decoding step reads the weight once and does next to nothing with it: HBM bounds it (11008 x 4096: 90 MB, 13.8 us at the
// measured copy bandwidth).  The CTA-pair GEMM (gemm_tc.cu) streams at that rate too but starts and ends in 5.5 us (barriers,
// tensor memory, clusters, tensor maps, staged stores).  Here every SM has one light block with an equal share of the rows, which
// come straight from global memory into registers, 16 to 24 vectors of 16 bytes ahead per thread (64 to 96 KB an SM), and into
// the warps' matrix instruction (m16n8k16): 2.6 us for start and end.  A warp takes every kWarps-th piece of 64 columns of
// all the block's rows.  The order of the columns inside a piece does not matter to a sum as long as both operands agree, so
// a lane's fragment of w is the 16 consecutive bytes it has loaded, of x likewise: nothing goes through shared memory, and x
// is read once by a block, which holds all its rows' sums.  The warps' sums meet in shared memory, in order, at the end.
//
// Measured (us, one layer called again and again; with three layers in turn 15.3 where the first figure is 16.4; weight settled, not
// settled / gemm_tc.cu) for 1, 8 and 16 tokens: 11008 x 4096 16.4 17.9 / 19.7, 16.8 18.2 / 19.8,
// 18.8 20.5 / 19.9; 4096 x 4096 8.0 9.3 / 10.0, 8.8 10.0 / 10.0, 9.7 10.7 / 10.0; 8192 x 1024 4.8 5.9 / 6.5, 5.3 6.3 / 6.5,
// 6.5 7.5 / 6.5; 2048 x 2048 4.3 / 5.7.  32 tokens would need more registers than there are (28.7 / 20.4).  Fused multiply-adds with x
// in shared memory instead: as fast for one token and long rows, 29.6 for 8 tokens at 11008 x 4096.
#include <algorithm>

#include "csr_terms.cuh"

namespace iex {
namespace tc {
namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kTileRows = 16;
constexpr int kMaxTiles = 6;     // row tiles of a block
constexpr int kPiece = 64;
constexpr int kMaxTokens = 16;

struct FewParams {
  int rows, k;
  const __half* w;
  long long ldw;
  const __half* x;
  long long ldx;
  int tokens;
  __half* out;
  long long ldo;
  int settled;  // nothing that may still run writes w: its first pieces are requested ahead of the wait
  CsrTerms terms;
};

// Read once by this SM.  Neither invariant nor ".nc": the kernel in front, which may still run when this one starts, can have
// written what is read, and loads that claim otherwise are moved ahead of a conditional grid_dependency_wait() (seen
// as wrong results of chained calls).
__device__ __forceinline__ uint4 load_once(const uint4* p) {
  uint4 v;
  asm volatile("ld.global.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p)
               : "memory");
  return v;
}

__device__ __forceinline__ void mma_16x8x16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                            uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// NT: groups of 8 tokens, MT: row tiles.  A block keeps kAheadPieces pieces of all its rows on their way.
template <int NT, int MT, bool kStored>
__global__ void __launch_bounds__(kThreads, 1) linear_few_mma_kernel(const __grid_constant__ FewParams p) {
  extern __shared__ float sums[];  // [kWarps][MT * 16][8 NT + 4]
  constexpr int kPitch = 8 * NT + 4, kAheadPieces = MT >= 5 ? 1 : MT >= 2 ? 2 : 4;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
  const int begin = static_cast<int>(static_cast<long long>(blockIdx.x) * p.rows / gridDim.x);
  const int end = static_cast<int>(static_cast<long long>(blockIdx.x + 1) * p.rows / gridDim.x);
  const int pieces = (p.k + kPiece - 1) / kPiece;

  struct Step { uint4 v[2][2]; };  // [row g, g + 8][first, second half of the piece]
  const uint4 none = make_uint4(0, 0, 0, 0);
  auto request = [&](Step& to, int piece, int tile) {
    const int row = begin + tile * kTileRows + g, c = piece * kPiece + q * 8;
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        to.v[r][h] = none;
        if (piece < pieces && row + 8 * r < end && c + 32 * h < p.k)
          to.v[r][h] = load_once(reinterpret_cast<const uint4*>(p.w + static_cast<size_t>(row + 8 * r) * p.ldw + c + 32 * h));
      }
  };
  auto fetch_x = [&](uint4 (&to)[NT][2], int piece) {
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int t = j * 8 + g, c = piece * kPiece + q * 8 + 32 * h;
        to[j][h] = none;
        if (piece < pieces && t < p.tokens && c < p.k) to[j][h] = load_once(reinterpret_cast<const uint4*>(p.x + t * p.ldx + c));
      }
  };
  Step w[kAheadPieces][MT];
  auto request_first = [&] {
#pragma unroll
    for (int u = 0; u < kAheadPieces; ++u)
#pragma unroll
      for (int i = 0; i < MT; ++i) request(w[u][i], warp + u * kWarps, i);
  };
  if (p.settled) request_first();
  grid_dependency_wait();
  if (!p.settled) request_first();
  uint4 x[NT][2], x_next[NT][2];
  fetch_x(x, warp);
  grid_launch_dependents();
  float acc[MT][NT][4];
#pragma unroll
  for (int i = 0; i < MT; ++i)
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.f;

  auto product = [&](float (&c)[NT][4], const Step& s) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint4 lo = s.v[0][h], hi = s.v[1][h];
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        mma_16x8x16(c[j], lo.x, hi.x, lo.y, hi.y, x[j][h].x, x[j][h].y);
        mma_16x8x16(c[j], lo.z, hi.z, lo.w, hi.w, x[j][h].z, x[j][h].w);
      }
    }
  };
  for (int first = warp; first < pieces; first += kAheadPieces * kWarps) {
#pragma unroll
    for (int u = 0; u < kAheadPieces; ++u) {
      const int piece = first + u * kWarps;
      fetch_x(x_next, piece + kWarps);
#pragma unroll
      for (int i = 0; i < MT; ++i) {
        product(acc[i], w[u][i]);
        request(w[u][i], piece + kAheadPieces * kWarps, i);
      }
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int h = 0; h < 2; ++h) x[j][h] = x_next[j][h];
    }
  }
  constexpr int lines = MT * kTileRows;
#pragma unroll
  for (int i = 0; i < MT; ++i)
#pragma unroll
    for (int j = 0; j < NT; ++j) {
      float* to = sums + (warp * lines + i * kTileRows + g) * kPitch + j * 8 + q * 2;
      *reinterpret_cast<float2*>(to) = make_float2(acc[i][j][0], acc[i][j][1]);
      *reinterpret_cast<float2*>(to + 8 * kPitch) = make_float2(acc[i][j][2], acc[i][j][3]);
    }
  __syncthreads();
  const int n = end - begin;
  for (int i = threadIdx.x; i < n * p.tokens; i += kThreads) {
    const int t = i / n, r = i - t * n;
    float sum = 0.f;
#pragma unroll
    for (int j = 0; j < kWarps; ++j) sum += sums[(j * lines + r) * kPitch + t];
    if (kStored && sum != sum) sum = sum_stored(p.terms, begin + r, t);
    p.out[t * p.ldo + begin + r] = __float2half_rn(sum);
  }
}

template <int NT, int MT>
int launch_mma(const FewParams& p, int blocks, bool stored, cudaStream_t stream) {
  constexpr int smem = kWarps * MT * kTileRows * (8 * NT + 4) * 4;
  auto kern = stored ? linear_few_mma_kernel<NT, MT, true> : linear_few_mma_kernel<NT, MT, false>;
  if constexpr (smem > 48 * 1024) {  // what a block may have without asking
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return static_cast<int>(e);
  }
  return launch_overlapped(kern, dim3(blocks), dim3(kThreads), static_cast<size_t>(smem), stream, p);
}

// A block per SM with an equal share of the rows; where that would be too many for a block's registers, two or more rounds.
template <int NT>
int launch(const FewParams& p, bool stored, cudaStream_t stream) {
  constexpr int most = kMaxTiles * kTileRows * kNumSMs;
  const int blocks = std::min((p.rows + 7) / 8, kNumSMs * ((p.rows + most - 1) / most));
  const int tiles = ((p.rows + blocks - 1) / blocks + kTileRows - 1) / kTileRows;
  if (tiles == 1) return launch_mma<NT, 1>(p, blocks, stored, stream);
  if (tiles == 2) return launch_mma<NT, 2>(p, blocks, stored, stream);
  if (tiles == 3) return launch_mma<NT, 3>(p, blocks, stored, stream);
  if (tiles <= 5) return launch_mma<NT, 5>(p, blocks, stored, stream);
  return launch_mma<NT, 6>(p, blocks, stored, stream);
}

}  // namespace

bool linear_few_supported(int tokens, int in_features) {
  return tokens >= 1 && tokens <= kMaxTokens && in_features > 0 && in_features % 8 == 0;
}

// Microseconds, fitted to 78 measurements (512 to 16384 rows, 512 to 11008 columns, 1 to 16 tokens, settled and not); 1e30 for
// what the kernel does not take.  A weight that is not settled costs the latency of its first loads on top (1.3 us).  Callers
// choose the GEMM where its estimate, which is 1 to 2 us above what small products take, is below 1.15 times this one: the
// slower way by 6 % at most in those.
double linear_few_us(int tokens, int in_features, int out_features, bool settled) {
  if (!linear_few_supported(tokens, in_features)) return 1e30;
  const int rounds = (out_features + kMaxTiles * kTileRows * kNumSMs - 1) / (kMaxTiles * kTileRows * kNumSMs);
  const double rate = tokens <= 8 ? 6.6e6 : settled ? 5.6e6 : 4.6e6;
  return (settled ? 2.6 : 3.9) + 2.0 * (rounds - 1) + std::max(1.6, 2.0 * out_features * in_features / rate);
}

// x, w and their rows on 16-byte boundaries.
int linear_few(int tokens, int in_features, int out_features, const void* x, long long ldx, const void* w, long long ldw,
               void* out, long long ldo, bool settled, const CsrTerms* terms, cudaStream_t stream) {
  if (!linear_few_supported(tokens, in_features) || ldx % 8 != 0 || ldw % 8 != 0 || !aligned16(x) || !aligned16(w))
    return IEX_ERR_UNSUPPORTED;
  if (out_features == 0) return IEX_OK;
  FewParams p{};
  p.rows = out_features;
  p.k = in_features;
  p.w = static_cast<const __half*>(w);
  p.ldw = ldw;
  p.x = static_cast<const __half*>(x);
  p.ldx = ldx;
  p.tokens = tokens;
  p.out = static_cast<__half*>(out);
  p.ldo = ldo;
  p.settled = settled;
  if (terms != nullptr) p.terms = *terms;
  const bool stored = terms != nullptr;
  return tokens <= 8 ? launch<1>(p, stored, stream) : launch<2>(p, stored, stream);
}

}  // namespace tc
}  // namespace iex

extern "C" int iex_linear_f16_few_supported(int tokens, int in_features) {
  return iex::tc::linear_few_supported(tokens, in_features) ? 1 : 0;
}

extern "C" double iex_linear_f16_few_estimate_us(int tokens, int in_features, int out_features, int weight_settled) {
  return iex::tc::linear_few_us(tokens, in_features, out_features, weight_settled != 0);
}

extern "C" int iex_linear_f16_few(int tokens, int in_features, int out_features, const void* input, const void* weight,
                                  void* out, int weight_settled, const int32_t* row_offsets, const void* column_indices,
                                  int index_bits, const void* values, void* stream) {
  if (tokens < 0 || in_features < 0 || out_features < 0) return IEX_ERR_BAD_ARG;
  if (tokens == 0 || out_features == 0) return IEX_OK;
  if (!input || !weight || !out) return IEX_ERR_BAD_ARG;
  if (row_offsets != nullptr && (!column_indices || !values || (index_bits != 16 && index_bits != 32))) return IEX_ERR_BAD_ARG;
  iex::tc::CsrTerms t{};
  t.row_offsets = row_offsets;
  t.cols = column_indices;
  t.values = static_cast<const __half*>(values);
  t.dense = static_cast<const __half*>(input);
  t.dense_c = 1;
  t.dense_t = in_features;
  t.rows = out_features;
  t.columns = tokens;
  t.index_bits = index_bits;
  return iex::tc::linear_few(tokens, in_features, out_features, input, in_features, weight, in_features, out, out_features,
                             weight_settled != 0, row_offsets ? &t : nullptr, static_cast<cudaStream_t>(stream));
}
