// Dense fp16 GEMM on CTA pairs (tcgen05 cta_group::2), fp32 accumulation, fp16 result:
//   D[m, n] = sum_k A(m, k) * B(n, k)
// A and B may each be stored with k contiguous ("K-major", [rows, K]) or with the row index
// contiguous ("MN-major", [K, rows]); D is written as [M, N] or transposed as [N, M].  That covers the
// dense branch's forward pass and both products of its backward pass without a transposed copy,
// and, with the weight as A and the activations as B, few-token inputs without padding the
// token dimension to 256.
//
// Decomposition.  Two CTAs of a cluster work on one 256 x bn tile of D: each keeps 128 rows of A
// and half of B's rows in shared memory and 128 rows of the accumulator in its tensor memory, so
// a k-block of 64 costs a CTA 16 KB of A and bn * 64 bytes of B instead of the bn * 128 that a CTA
// working alone would load: the L2 -> SM path, not the tensor pipe, bounds the one-CTA kernel of
// tc_fused.cu (256 x 11008 -> 4096: 270 MB through it for 96 MB of operands).  bn is a run-time
// multiple of 32 up to 256, chosen so that the tiles fill the last wave (plan_gemm).
//
//   warp 0     TMA producer (both CTAs): own halves of A and B, completion on the leader's barrier
//   warp 1     MMA issuer (leader CTA): tcgen05.mma M256 x bn x K16, commits to both CTAs
//   warps 2-5  epilogue: tcgen05.ld, fp16, 4 KB staging per warp, TMA store
// Two accumulators of 256 columns alternate, so a tile's epilogue runs under the next tile's
// main loop.  When there are too few tiles for the chip, a cluster of 2 * P CTAs splits K over
// its P pairs and adds the fp32 partial tiles through distributed shared memory, in part order
// (deterministic, no workspace and no second launch).
//
// Measured against the one-CTA kernel: 2048 x 4096 -> 12288, forward and backward, 1245 -> 452-520 us (the power limit
// moves it; the three products alone 146 / 148 / 144 us, 1.41 PFLOP/s); 256 x 11008 -> 4096 35.3 -> 26.1 us; 64 x 4096 ->
// 12288 23.4 us, where HBM bounds both.
//
// Every mbarrier wait is bounded, as in tc_fused.cu.
#include <cuda.h>

#include <algorithm>
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

constexpr int kBK = 64;                    // k per stage: one 128-byte swizzle atom
constexpr int kHalfM = 128;                // rows of A per CTA
constexpr int kABytes = kHalfM * 128;      // one stage of A
constexpr int kMaxStages = 9;
constexpr int kThreads = 192;
constexpr int kStagingBytes = 4 * 2 * 4096;  // per epilogue warp two 4 KB buffers
constexpr int kAccumCols = 256;            // columns between the two accumulators
constexpr int kBarBytes = 8 * (2 * kMaxStages + 4) + 16;
constexpr int kSmemBudget = 227 * 1024 - 1024 - kBarBytes;

struct GemmParams {
  int m, n, k;
  int bn;                  // tile columns
  int tiles_m, tiles_n;
  int stages;
  int parts;               // pairs of a cluster that split K (1: persistent, no split)
  int out_t;
  int tma_out;             // rows of the output are multiples of 16 bytes: TMA stores
  __half* out;
  long long ldo;           // elements between rows of the stored output
  CsrTerms terms;          // kStored: one operand is the dense copy of this CSR matrix
  int* status;
};

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t map_to_rank(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// TMA load into this CTA's shared memory whose bytes are counted on a barrier of the pair
__device__ __forceinline__ void tma_load_pair(uint32_t dst, const CUtensorMap* map, uint32_t cluster_bar, int c0,
                                              int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4}], [%2];" ::"r"(dst),
      "l"(map), "r"(cluster_bar), "r"(c0), "r"(c1)
      : "memory");
}
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, uint32_t src, int c0, int c1) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(map), "r"(src),
               "r"(c0), "r"(c1)
               : "memory");
}
__device__ __forceinline__ void umma_f16_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                              uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// arrives, when all MMAs issued before have completed, on the barrier at this offset in every CTA of `mask`
__device__ __forceinline__ void umma_commit_pair(uint32_t bar, uint16_t mask) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
      "h"(mask)
      : "memory");
}

// Tile order: groups of 8 tile rows, columns inside a group, so that the tiles in flight share
// both operands in L2.
__device__ __forceinline__ void tile_of(int t, const GemmParams& p, int& tm, int& tn) {
  constexpr int kGroup = 8;
  const int per_group = kGroup * p.tiles_n;
  const int g = t / per_group, first = g * kGroup;
  const int rows = min(kGroup, p.tiles_m - first);
  const int r = t - g * per_group;
  tm = first + r % rows;
  tn = r / rows;
}

// Sums of the P partial tiles of a cluster, in part order, from the CTAs' shared memory.  A load from another CTA takes
// about 0.4 us and this is all that is left to do, so a thread keeps 8 to 12 of them in flight: with one vector at a time
// the
// exchange of a 256 x 256 tile between two pairs took 8 us, now 3 us (256 x 4096 x 11008: 39.5 -> 34.4 us, with 128-wide
// tiles 27.2 -> 25.2 us).
template <int P, typename Write>
__device__ __forceinline__ void add_parts(uint32_t base, int l0, int vecs, uint32_t vec_inv, uint32_t line_bytes, int total,
                                          int half, const Write& write) {
  constexpr int U = P == 2 ? 6 : P == 3 ? 4 : 3;
  for (int f0 = threadIdx.x; f0 < total; f0 += U * kThreads) {
    float4 x[U][P];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int f = min(f0 + u * kThreads, total - 1);
      const uint32_t line = (static_cast<uint32_t>(f) * vec_inv) >> 20;
      const uint32_t off = base + (l0 + line) * line_bytes + (f - line * vecs) * 16u;
#pragma unroll
      for (int q = 0; q < P; ++q)
        asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                     : "=f"(x[u][q].x), "=f"(x[u][q].y), "=f"(x[u][q].z), "=f"(x[u][q].w)
                     : "r"(map_to_rank(off, 2 * q + half)));
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      float4 sum = x[u][0];
#pragma unroll
      for (int q = 1; q < P; ++q) {
        sum.x += x[u][q].x; sum.y += x[u][q].y; sum.z += x[u][q].z; sum.w += x[u][q].w;
      }
      if (f0 + u * kThreads < total) write(f0 + u * kThreads, sum);
    }
  }
}

// A warp's 32 rows of a tile, from tensor memory to the output, 32 rows x 32 columns at a time.  kSum: returns the sum of what
// the thread has read, NaN if any of it is.  kRepair: NaN outputs are summed from the stored positions (csr_terms.cuh).
template <bool kSum, bool kRepair>
__device__ __forceinline__ float store_tile(const GemmParams& p, const CUtensorMap& map_out, uint32_t taddr, uint32_t stage0,
                                            int& buf, int row0, int tn, int lane) {
  float sum = 0.f;
  const int cols = min(p.bn, p.n - tn * p.bn);
  for (int c = 0; c < cols; c += 64) {
    // a buffer is written again only when its earlier store has read it
    if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
    __syncwarp();
    const uint32_t dst = stage0 + buf * 4096u;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (c + h * 32 >= p.bn) break;
      uint32_t r[32];
      tmem_ld32(taddr + c + h * 32, r);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      if constexpr (kSum) sum += sum_words(r);
      if constexpr (kRepair) {
        const int row = row0 + lane, col = tn * p.bn + c + h * 32;
        if (p.terms.sparse_is_a) repair(p.terms, row, col, 0, 1, r);
        else repair(p.terms, col, row, 1, 0, r);
        __syncwarp();
      }
      if (p.out_t) {  // [N, M]: 32 columns of D x 64 bytes of rows
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          const uint16_t hv = __half_as_ushort(__float2half_rn(__uint_as_float(r[j])));
          asm volatile("st.shared.u16 [%0], %1;" ::"r"(dst + h * 2048u + j * 64u + lane * 2u), "h"(hv) : "memory");
        }
      } else {        // [M, N]: 32 rows x 128 bytes, 128-byte swizzle
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          uint32_t w[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const __half2 hh = __floats2half2_rn(__uint_as_float(r[8 * j + 2 * e]), __uint_as_float(r[8 * j + 2 * e + 1]));
            w[e] = *reinterpret_cast<const uint32_t*>(&hh);
          }
          const uint32_t chunk = static_cast<uint32_t>(h * 4 + j) ^ (lane & 7u);
          asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(dst + lane * 128u + chunk * 16u), "r"(w[0]),
                       "r"(w[1]), "r"(w[2]), "r"(w[3])
                       : "memory");
        }
      }
    }
    if (!p.tma_out) {  // rows of any length and alignment ([M, N] only): two-byte stores, coalesced
      __syncwarp();
      const int n_left = cols - c;
      for (int i = lane; i < 32 * 64; i += 32) {
        const int rr = i >> 6, cc = i & 63;
        if (row0 + rr < p.m && cc < n_left) {
          const uint32_t chunk = static_cast<uint32_t>(cc >> 3) ^ (rr & 7u);
          uint16_t hv;
          asm volatile("ld.shared.u16 %0, [%1];" : "=h"(hv) : "r"(dst + rr * 128u + chunk * 16u + (cc & 7) * 2u));
          p.out[static_cast<size_t>(row0 + rr) * p.ldo + tn * p.bn + c + cc] = __ushort_as_half(hv);
        }
      }
      __syncwarp();
      continue;
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
    if (lane == 0) {
      const int col0 = tn * p.bn + c;
      if (row0 < p.m) {
        if (p.out_t) {
          tma_store_2d(&map_out, dst, row0, col0);
          if (c + 32 < cols) tma_store_2d(&map_out, dst + 2048u, row0, col0 + 32);
        } else {
          tma_store_2d(&map_out, dst, col0, row0);
        }
      }
      asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    }
    buf ^= 1;
  }
  return sum;
}

// Over what is there already.  A whole tile at a time and out of line: looking at every piece as it is read costs a tile 0.3
// us (8696 x 1408 x 479: 13.6 us, so 13.1, without any check 12.8).
__device__ __noinline__ void store_tile_again(const GemmParams& p, const CUtensorMap& map_out, uint32_t taddr, uint32_t stage0,
                                              int buf, int row0, int tn, int lane) {
  if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  __syncwarp();
  store_tile<false, true>(p, map_out, taddr, stage0, buf, row0, tn, lane);
  if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  __syncwarp();
}

// The operands' storage orders are template parameters for the sake of the one thread that issues the
// MMAs: its descriptors then advance by constants.  kStored: p.terms says which CSR matrix an operand is the dense copy of
// (a parameter too, since the path that sums outputs again costs every launch 0.2 us, by its registers and stack).
template <bool kAMn, bool kBMn, bool kStored>
__global__ void __launch_bounds__(kThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                 const __grid_constant__ CUtensorMap map_out, const __grid_constant__ GemmParams p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* base_ptr = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t b_bytes = kBMn ? ((p.bn / 2 + 63) / 64) * (kBK * 128u) : static_cast<uint32_t>(p.bn / 2) * 128u;
  const uint32_t stage_bytes = kABytes + b_bytes;
  const int S = p.stages;
  // data (stages; the partial tile of a split overlays them) | staging | barriers
  const uint32_t bar_off = kSmemBudget & ~15u;
  const uint32_t staging = base + ((bar_off - kStagingBytes) & ~1023u);
  const uint32_t bar = base + bar_off;
  auto full_bar = [&](int s) { return bar + 8u * s; };
  auto empty_bar = [&](int s) { return bar + 8u * (kMaxStages + s); };
  auto acc_full = [&](int a) { return bar + 8u * (2 * kMaxStages + a); };
  auto acc_empty = [&](int a) { return bar + 8u * (2 * kMaxStages + 2 + a); };
  const uint32_t tmem_slot = bar + 8u * (2 * kMaxStages + 4);
  volatile uint32_t* tmem_ptr = reinterpret_cast<volatile uint32_t*>(base_ptr + bar_off + 8u * (2 * kMaxStages + 4));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_ptr + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  const int half = rank & 1;                 // this CTA's half of the tile's rows
  const int part = static_cast<int>(rank >> 1);
  const uint32_t leader = rank & ~1u;
  const int cluster_size = 2 * p.parts;
  const int unit0 = static_cast<int>(blockIdx.x) / cluster_size, unit_step = static_cast<int>(gridDim.x) / cluster_size;
  const int tiles = p.tiles_m * p.tiles_n;
  const int k_blocks = (p.k + kBK - 1) / kBK;
  const int kb0 = part * k_blocks / p.parts, kb1 = (part + 1) * k_blocks / p.parts;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kMaxStages; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(acc_full(a), 1);
      mbar_init(acc_empty(a), 8);  // four epilogue warps in each of the two CTAs
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_slot), "r"(512u)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tcgen05_fence_before();
  __syncthreads();
  cluster_sync_all();  // barriers of both CTAs exist before either signals the other
  tcgen05_fence_after();
  const uint32_t tmem = *tmem_ptr;
  grid_dependency_wait();
  grid_launch_dependents();

  if (warp == 0) {
    if (elect_one()) {
      asm volatile("prefetch.tensormap [%0];" ::"l"(&map_a) : "memory");
      asm volatile("prefetch.tensormap [%0];" ::"l"(&map_b) : "memory");
      asm volatile("prefetch.tensormap [%0];" ::"l"(&map_out) : "memory");
      bool ok = true;
      int s = 0;
      uint32_t ph = 0;
      for (int t = unit0; t < tiles && ok; t += unit_step) {
        int tm, tn;
        tile_of(t, p, tm, tn);
        const int row_a = tm * 256 + half * kHalfM;
        const int row_b = tn * p.bn + half * (p.bn / 2);
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait(empty_bar(s), ph ^ 1u, abort_flag, p.status, 32)) { ok = false; break; }
          const uint32_t a_dst = base + s * stage_bytes, b_dst = a_dst + kABytes;
          const uint32_t fb = map_to_rank(full_bar(s), leader);
          if (half == 0) mbar_arrive_expect_tx(full_bar(s), 2u * stage_bytes);
          if (kAMn) {  // [K, M]: two boxes of 64 k-rows x 64 columns
            tma_load_pair(a_dst, &map_a, fb, row_a, kb * kBK);
            tma_load_pair(a_dst + kBK * 128, &map_a, fb, row_a + 64, kb * kBK);
          } else {       // [M, K]: one box of 128 rows x 64 k
            tma_load_pair(a_dst, &map_a, fb, kb * kBK, row_a);
          }
          if (kBMn) {
            for (int j = 0; j < (p.bn / 2 + 63) / 64; ++j)
              tma_load_pair(b_dst + j * (kBK * 128), &map_b, fb, row_b + j * 64, kb * kBK);
          } else {
            tma_load_pair(b_dst, &map_b, fb, kb * kBK, row_b);
          }
          if (++s == S) { s = 0; ph ^= 1u; }
        }
      }
      if (!ok)  // drain: bounded time for the copies this thread armed to land
        for (uint32_t i = 0; i < 2048u; ++i) __nanosleep(100);
    }
    __syncwarp();
  } else if (warp == 1) {
    if (half == 0 && elect_one()) {
      const uint32_t idesc = (1u << 4) | (kAMn ? (1u << 15) : 0u) | (kBMn ? (1u << 16) : 0u) |
                             (static_cast<uint32_t>(p.bn >> 3) << 17) | (16u << 24);
      const uint16_t mask = static_cast<uint16_t>(3u << leader);
      constexpr uint32_t a_step = kAMn ? 16u * 128u : 32u, b_step = kBMn ? 16u * 128u : 32u;  // K16 further
      bool ok = true;
      int s = 0, u = 0;
      uint32_t ph = 0;
      for (int t = unit0; t < tiles && ok; t += unit_step, ++u) {
        const int acc = u & 1;
        // an accumulator whose outputs are summed again (csr_terms.cuh) may take tens of ms to read out
        if (!mbar_wait(acc_empty(acc), ((u >> 1) & 1u) ^ 1u, abort_flag, p.status, 32, kStored ? 1024 : 0)) {
          ok = false;
          break;
        }
        tcgen05_fence_after();
        const uint32_t d = tmem + acc * kAccumCols;
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait(full_bar(s), ph, abort_flag, p.status, 32)) { ok = false; break; }
          tcgen05_fence_after();
          const uint32_t a_addr = base + s * stage_bytes;
          const uint64_t ad = kAMn ? smem_desc(a_addr, kBK * 128, 1024) : smem_desc(a_addr, 16, 1024);
          const uint64_t bd = kBMn ? smem_desc(a_addr + kABytes, kBK * 128, 1024) : smem_desc(a_addr + kABytes, 16, 1024);
#pragma unroll
          for (int ks = 0; ks < kBK / 16; ++ks)
            umma_f16_pair(d, desc_advance(ad, ks * a_step), desc_advance(bd, ks * b_step), idesc,
                          (kb != kb0 || ks != 0) ? 1u : 0u);
          umma_commit_pair(empty_bar(s), mask);
          if (++s == S) { s = 0; ph ^= 1u; }
        }
        if (ok) umma_commit_pair(acc_full(acc), mask);
      }
    }
    __syncwarp();
  } else if (p.parts == 1) {
    // ---- epilogue of whole tiles: 32 rows x 32 columns at a time
    const int q = warp & 3;
    const uint32_t stage0 = staging + (warp - 2) * 8192u;
    int u = 0, buf = 0;
    for (int t = unit0; t < tiles; t += unit_step, ++u) {
      const int acc = u & 1;
      int tm, tn;
      tile_of(t, p, tm, tn);
      if (!mbar_wait(acc_full(acc), (u >> 1) & 1u, abort_flag, p.status, 64)) break;
      tcgen05_fence_after();
      const int row0 = tm * 256 + half * kHalfM + q * 32;
      const uint32_t taddr = tmem + acc * kAccumCols + (static_cast<uint32_t>(q * 32) << 16);
      const float sum = store_tile<kStored, false>(p, map_out, taddr, stage0, buf, row0, tn, lane);
      if constexpr (kStored) {
        if (__any_sync(0xffffffffu, sum != sum)) store_tile_again(p, map_out, taddr, stage0, buf, row0, tn, lane);
      }
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(map_to_rank(acc_empty(acc), leader));
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    __syncwarp();
  } else {
    // ---- split K: this pair's fp32 partial tile into shared memory (over the stages)
    const int q = warp & 3;
    if (mbar_wait(acc_full(0), 0, abort_flag, p.status, 64)) {
      tcgen05_fence_after();
      const uint32_t taddr = tmem + (static_cast<uint32_t>(q * 32) << 16);
      const int row = q * 32 + lane;
      for (int c = 0; c < p.bn; c += 32) {
        uint32_t r[32];
        tmem_ld32(taddr + c, r);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (p.out_t) {  // [bn][128]
#pragma unroll
          for (int j = 0; j < 32; ++j)
            asm volatile("st.shared.u32 [%0], %1;" ::"r"(base + ((c + j) * kHalfM + row) * 4u), "r"(r[j]) : "memory");
        } else {        // [128][bn + 4]
#pragma unroll
          for (int j = 0; j < 8; ++j)
            asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(base + (row * (p.bn + 4) + c + 4 * j) * 4u),
                         "r"(r[4 * j]), "r"(r[4 * j + 1]), "r"(r[4 * j + 2]), "r"(r[4 * j + 3])
                         : "memory");
        }
      }
      tcgen05_fence_before();
    }
  }
  if (p.parts > 1) {
    __syncwarp();
    cluster_sync_all();
    // CTA `part` of a half adds columns (out_t) or rows of the P partial tiles and writes them
    int tm, tn;
    tile_of(unit0, p, tm, tn);
    const int row0 = tm * 256 + half * kHalfM, col0 = tn * p.bn;
    const int vecs = p.out_t ? kHalfM / 4 : p.bn / 4;            // float4 per line
    const int lines = p.out_t ? p.bn : kHalfM;                   // lines of the partial tile
    const uint32_t line_bytes = (p.out_t ? kHalfM : p.bn + 4) * 4u;
    const int l0 = part * lines / p.parts, l1 = (part + 1) * lines / p.parts;
    const uint32_t vec_inv = ((1u << 20) + vecs - 1) / vecs;  // f / vecs: f is below 4096, vecs 8 to 64
    auto write = [&](int f, const float4& total) {
      const int line = l0 + static_cast<int>((static_cast<uint32_t>(f) * vec_inv) >> 20);
      const int v = f - (line - l0) * vecs;
      float4 sum = total;
      if constexpr (kStored) {
        uint32_t r[4] = {__float_as_uint(sum.x), __float_as_uint(sum.y), __float_as_uint(sum.z), __float_as_uint(sum.w)};
        const int row = row0 + (p.out_t ? v * 4 : line), col = col0 + (p.out_t ? line : v * 4);
        const int row_step = p.out_t ? 1 : 0;
        if (p.terms.sparse_is_a) repair(p.terms, row, col, row_step, 1 - row_step, r);
        else repair(p.terms, col, row, 1 - row_step, row_step, r);
        sum = make_float4(__uint_as_float(r[0]), __uint_as_float(r[1]), __uint_as_float(r[2]), __uint_as_float(r[3]));
      }
      uint2 pk;
      __half2* hh = reinterpret_cast<__half2*>(&pk);
      hh[0] = __floats2half2_rn(sum.x, sum.y);
      hh[1] = __floats2half2_rn(sum.z, sum.w);
      const int outer = p.out_t ? col0 + line : row0 + line;
      const int inner = (p.out_t ? row0 : col0) + v * 4;
      const int n_outer = p.out_t ? p.n : p.m, n_inner = p.out_t ? p.m : p.n;
      if (outer < n_outer && inner < n_inner) {
        __half* dst = p.out + static_cast<size_t>(outer) * p.ldo + inner;
        if (p.tma_out) {  // the contiguous dimension is a multiple of 8: a vector is inside or outside
          *reinterpret_cast<uint2*>(dst) = pk;
        } else {
          const __half* hv = reinterpret_cast<const __half*>(&pk);
          for (int e = 0; e < 4 && inner + e < n_inner; ++e) dst[e] = hv[e];
        }
      }
    };
    const int total = (l1 - l0) * vecs;
    if (p.parts == 2) add_parts<2>(base, l0, vecs, vec_inv, line_bytes, total, half, write);
    else if (p.parts == 3) add_parts<3>(base, l0, vecs, vec_inv, line_bytes, total, half, write);
    else add_parts<4>(base, l0, vecs, vec_inv, line_bytes, total, half, write);
  }
  // nobody leaves while the other CTAs may still read its shared memory or write its tensor memory
  tcgen05_fence_before();
  __syncthreads();
  cluster_sync_all();
  if (warp == 1) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
}

struct GemmPlan {
  int bn, parts;
};

int stages_for(int bn, bool b_mn) {
  const int b = b_mn ? ((bn / 2 + 63) / 64) * kBK * 128 : bn / 2 * 128;
  const int data = (kSmemBudget & ~15) - kStagingBytes - 1024;
  const int s = data / (kABytes + b);
  return s > kMaxStages ? kMaxStages : s;
}

// Clusters of 2 * parts CTAs (one CTA per SM) that a B200 holds at a time: the SMs of a cluster
// belong to one GPC, so large clusters leave some SMs out.
constexpr int kResident[5] = {0, 74, 33, 22, 15};

// Tile width and K split for the smallest estimated time, in microseconds.  Fitted to a sweep over shapes on B200,
// within about 5 %: a k-block takes 0.155 us + 0.0001 us per tile column, or 0.00118 us per column where the tensor pipe bounds
// it (from 144 columns), or what L2 delivers to all CTAs together (17.5 TB/s); rows of B that run along n cost 0.02 us
// more.  HBM gives 5.8 TB/s; where the two bounds are close they add up rather than hide each other.  A launch has
// 5.3 us of its own (first loads, read-out), an exchange between the parts 0.3 us and 0.0095 us per column.
double plan_gemm(int m, int n, int k, bool b_mn, bool out_t, int sms, GemmPlan* plan) {
  const int kb = (k + kBK - 1) / kBK, tm = (m + 255) / 256;
  const double dram = (static_cast<double>(m) * k + static_cast<double>(n) * k + static_cast<double>(m) * n) * 2.0 / 5.8e6;
  double best = 1e30;
  for (int bn = 256; bn >= 32; bn -= 32) {
    if ((b_mn || !out_t) && bn % 64 != 0) continue;  // 64-column atoms / output boxes
    if (bn >= n + 64) continue;                      // columns nobody asked for
    const int tiles = tm * ((n + bn - 1) / bn);
    const double alone = std::max(0.155 + 0.0001 * bn, 0.00118 * bn) + (b_mn ? 0.02 : 0.0);
    for (int parts = 1; parts <= 4; ++parts) {
      const int resident = parts == 1 ? sms / 2 : kResident[parts];
      if (parts > 1 && (tiles > resident || kb < 4 * parts)) continue;
      const int waves = (tiles + resident - 1) / resident;
      const int ctas = 2 * parts * std::min(tiles, resident);
      const double block = std::max(alone, ctas * (kABytes + 64.0 * bn) / 17.5e6);
      const double loop = waves * ((kb + parts - 1) / parts * block + 0.3);
      const double l2 = loop * loop, d2 = dram * dram;
      const double t = std::sqrt(std::sqrt(l2 * l2 + d2 * d2)) + 5.0 + 0.5 * bn / 256 + (parts > 1 ? 0.3 + 0.0095 * bn : 0.0);
      if (t < best) { best = t; *plan = {bn, parts}; }
    }
  }
  return best;
}

}  // namespace

// lda, ldb, ldo: elements between consecutive rows of the stored arrays (multiples of 8 for the
// operands; any for a row-major output).
int gemm_f16(int m, int n, int k, const void* a, bool a_mn, long long lda, const void* b, bool b_mn, long long ldb,
             void* out, bool out_t, long long ldo, int force_bn, int force_parts, cudaStream_t stream,
             const CsrTerms* terms = nullptr) {
  if (m < 0 || n < 0 || k < 0) return IEX_ERR_BAD_ARG;
  if (m == 0 || n == 0) return IEX_OK;
  if (!out || (k > 0 && (!a || !b))) return IEX_ERR_BAD_ARG;
  if (lda < (a_mn ? m : k) || ldb < (b_mn ? n : k) || ldo < (out_t ? m : n)) return IEX_ERR_BAD_ARG;
  if (k == 0 || lda % 8 != 0 || ldb % 8 != 0 || !aligned16(a) || !aligned16(b))
    return IEX_ERR_UNSUPPORTED;  // rows of a tensor map are multiples of 16 bytes
  const bool tma_out = (out_t ? m : n) % 8 == 0 && ldo % 8 == 0 && aligned16(out);
  if (out_t && !tma_out) return IEX_ERR_UNSUPPORTED;
  const int sms = sm_count();
  GemmPlan plan{};
  if (force_bn <= 0 || force_parts <= 0) plan_gemm(m, n, k, b_mn, out_t, sms, &plan);
  if (force_bn > 0) plan.bn = force_bn;
  if (force_parts > 0) plan.parts = force_parts;
  if (plan.bn % (b_mn || !out_t ? 64 : 32) != 0 || plan.bn > 256 || plan.bn <= 0) return IEX_ERR_BAD_ARG;
  if (plan.parts < 1 || plan.parts > 4 || plan.parts > (k + kBK - 1) / kBK) return IEX_ERR_BAD_ARG;
  CUtensorMap ma, mb, mo;
  int st = a_mn ? make_map_f16(&ma, a, k, m, lda, kBK, 64, true) : make_map_f16(&ma, a, m, k, lda, kHalfM, 64, true);
  if (st == IEX_OK)
    st = b_mn ? make_map_f16(&mb, b, k, n, ldb, kBK, 64, true) : make_map_f16(&mb, b, n, k, ldb, plan.bn / 2, 64, true);
  if (st == IEX_OK && tma_out)
    st = out_t ? make_map_f16(&mo, out, n, m, ldo, 32, 32, false) : make_map_f16(&mo, out, m, n, ldo, 32, 64, true);
  if (st != IEX_OK) return st;
  if (!tma_out) mo = ma;  // not used
  GemmParams p{};
  p.m = m; p.n = n; p.k = k;
  p.bn = plan.bn;
  p.tiles_m = (m + 255) / 256;
  p.tiles_n = (n + plan.bn - 1) / plan.bn;
  p.stages = stages_for(plan.bn, b_mn);
  p.parts = plan.parts;
  p.out_t = out_t;
  p.tma_out = tma_out;
  p.out = static_cast<__half*>(out);
  p.ldo = ldo;
  if (terms != nullptr) p.terms = *terms;
  p.status = status_word();
  constexpr size_t smem = 227 * 1024;
  auto kern = terms == nullptr ? (a_mn ? (b_mn ? gemm_pair_kernel<true, true, false> : gemm_pair_kernel<true, false, false>)
                                       : (b_mn ? gemm_pair_kernel<false, true, false> : gemm_pair_kernel<false, false, false>))
                               : (a_mn ? (b_mn ? gemm_pair_kernel<true, true, true> : gemm_pair_kernel<true, false, true>)
                                       : (b_mn ? gemm_pair_kernel<false, true, true> : gemm_pair_kernel<false, false, true>));
  {
    static std::mutex mutex;
    static bool configured[64][8] = {};
    const int which = (terms ? 4 : 0) + (a_mn ? 2 : 0) + (b_mn ? 1 : 0);
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) dev = -1;
    std::lock_guard<std::mutex> lock(mutex);
    if (dev < 0 || dev >= 64 || !configured[dev][which]) {
      const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
      if (e != cudaSuccess) return static_cast<int>(e);
      if (dev >= 0 && dev < 64) configured[dev][which] = true;
    }
  }
  const int tiles = p.tiles_m * p.tiles_n;
  const int cluster = 2 * plan.parts;
  const int units = plan.parts > 1 ? tiles : (tiles < sms / 2 ? tiles : sms / 2);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(units * cluster);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cluster;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, ma, mb, mo, p);
  return static_cast<int>(e != cudaSuccess ? e : cudaGetLastError());
}

int linear_few(int tokens, int in_features, int out_features, const void* x, long long ldx, const void* w, long long ldw,
               void* out, long long ldo, bool settled, const CsrTerms* terms, cudaStream_t stream);  // linear_few.cu
double linear_few_us(int tokens, int in_features, int out_features, bool settled);

// The weight can be A (256-row tiles of features, the tokens as tile columns, result transposed) or
// B (tiles of 256 tokens): few tokens want the former, many the latter; whichever the estimate favours.
bool weight_as_a(int tokens, int features, int k, bool w_mn) {
  GemmPlan p{};
  const int sms = sm_count();
  return plan_gemm(features, tokens, k, false, true, sms, &p) <= plan_gemm(tokens, features, k, w_mn, false, sms, &p);
}

}  // namespace tc
}  // namespace iex

extern "C" int iex_gemm_f16(int m, int n, int k, const void* a, int a_mn, long long lda, const void* b, int b_mn,
                            long long ldb, void* out, int out_transposed, long long ldo, int tile_n, int k_parts,
                            void* stream) {
  return iex::tc::gemm_f16(m, n, k, a, a_mn != 0, lda, b, b_mn != 0, ldb, out, out_transposed != 0, ldo, tile_n,
                           k_parts, static_cast<cudaStream_t>(stream));
}

extern "C" int iex_gemm_f16_csr(int m, int n, int k, const void* a, int a_mn, long long lda, const void* b, int b_mn,
                                long long ldb, void* out, int out_transposed, long long ldo, int sparse_operand,
                                const int32_t* row_offsets, const void* column_indices, int index_bits, const void* values,
                                const long long* perm, int tile_n, int k_parts, void* stream) {
  if (sparse_operand < 0 || sparse_operand > 1 || (index_bits != 16 && index_bits != 32)) return IEX_ERR_BAD_ARG;
  if (m > 0 && n > 0 && (!row_offsets || (k > 0 && (!column_indices || !values)))) return IEX_ERR_BAD_ARG;
  iex::tc::CsrTerms t{};
  t.row_offsets = row_offsets;
  t.cols = column_indices;
  t.values = static_cast<const __half*>(values);
  t.perm = perm;
  t.index_bits = index_bits;
  t.sparse_is_a = sparse_operand == 0;
  t.rows = t.sparse_is_a ? m : n;
  t.columns = t.sparse_is_a ? n : m;
  // the other operand: its k dimension runs along rows (strides 1, ld) or down them (ld, 1)
  t.dense = static_cast<const __half*>(t.sparse_is_a ? b : a);
  const bool mn = (t.sparse_is_a ? b_mn : a_mn) != 0;
  const long long ld = t.sparse_is_a ? ldb : lda;
  t.dense_c = mn ? ld : 1;
  t.dense_t = mn ? 1 : ld;
  return iex::tc::gemm_f16(m, n, k, a, a_mn != 0, lda, b, b_mn != 0, ldb, out, out_transposed != 0, ldo, tile_n, k_parts,
                           static_cast<cudaStream_t>(stream), &t);
}

extern "C" double iex_gemm_f16_estimate_us(int m, int n, int k, int b_mn, int out_transposed) {
  iex::tc::GemmPlan plan{};
  return iex::tc::plan_gemm(m, n, k, b_mn != 0, out_transposed != 0, iex::tc::sm_count(), &plan);
}

// The dense branch, any number of tokens:
//   forward  out [tokens, out]     = input [tokens, in] * weight [out, in]^T
//   dgrad    dinput [tokens, in]   = grad [tokens, out] * weight [out, in]
//   wgrad    dweight [out, in]     = grad^T [out, tokens] * input [tokens, in]
// (layers_and_funcs/torch.py:17, :24-27), every operand read as it lies.
extern "C" int iex_linear_f16_any(int tokens, int in_features, int out_features, const void* input,
                                  const void* weight, void* out, void* stream) {
  using namespace iex::tc;
  const int t = tokens, i = in_features, o = out_features;
  const cudaStream_t s = static_cast<cudaStream_t>(stream);
  GemmPlan plan{}, rows_plan{};
  // the weight as A writes the result transposed, by TMA
  double gemm_us = o % 8 == 0 && iex::aligned16(out) ? plan_gemm(o, t, i, false, true, sm_count(), &plan) : 1e30;
  const double rows_us = plan_gemm(t, o, i, false, false, sm_count(), &rows_plan);
  const bool as_a = gemm_us <= rows_us;
  if (!as_a) gemm_us = rows_us;
  if (t > 0 && o > 0 && 1.15 * linear_few_us(t, i, o, false) <= gemm_us && input && weight && out && iex::aligned16(input) &&
      iex::aligned16(weight))
    return linear_few(t, i, o, input, i, weight, i, out, o, false, nullptr, s);  // a handful of tokens
  if (as_a) return gemm_f16(o, t, i, weight, false, i, input, false, i, out, true, o, plan.bn, plan.parts, s);
  return gemm_f16(t, o, i, input, false, i, weight, false, i, out, false, o, rows_plan.bn, rows_plan.parts, s);
}

extern "C" int iex_linear_f16_dgrad(int tokens, int in_features, int out_features, const void* grad,
                                    const void* weight, void* dinput, void* stream) {
  using namespace iex::tc;
  const int t = tokens, i = in_features, o = out_features;
  const cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (i % 8 == 0 && iex::aligned16(dinput) && weight_as_a(t, i, o, true))
    return gemm_f16(i, t, o, weight, true, i, grad, false, o, dinput, true, i, 0, 0, s);
  return gemm_f16(t, i, o, grad, false, o, weight, true, i, dinput, false, i, 0, 0, s);
}

extern "C" int iex_linear_f16_wgrad(int tokens, int in_features, int out_features, const void* grad,
                                    const void* input, void* dweight, void* stream) {
  return iex::tc::gemm_f16(out_features, in_features, tokens, grad, true, out_features, input, true, in_features,
                           dweight, false, in_features, 0, 0, static_cast<cudaStream_t>(stream));
}
