// GEMM core for products with too few output tiles to fill the GPU: one 128 x 128 (or 128 x 64) tile per cluster of S
// CTAs, each of which takes a share of K (bf16, or e4m3 with 1 x 128 / 128 x 128 block scales as in gemm_fp8_core.cuh).
//
// What bounds such a product is how many SMs read the weight: the persistent kernels give it one CTA per 256 columns,
// i.e. 28 of 148 SMs for 32 x 7168 x 8192 and 8 for 64 x 2048 x 7168 e4m3. Here every CTA leaves its fp32 partial tile
// in its own shared memory (over the ring, which is idle by then), the cluster synchronises, and CTA r adds up and
// stores every S-th part of the tile through distributed shared memory: no workspace in global memory, no counter, and
// the order of the sum is fixed. A single row block loads only the rows of A that exist (the box is cut to the next
// multiple of eight).
//
// Measured in a loop: 32 x 7168 x 8192 bf16 55.3 -> 28.3 us (4.2 TB/s; what is left is the rate at which 112 SMs read),
// 256 x 4096 x 4096 26.7 -> 19.7, 600 x 1500 x 4096 34.9 -> 18.9; 64 x 2048 x 7168 e4m3 33.0 -> 13.0 us (the host needs 10
// for a call), 200 x 2048 x 7168 36.0 -> 18.3.
//
//   warp 0      TMA producer, a ring of 128-byte K slabs of A and B;
//   warp 1      MMA issuer (M 128, N 128 or 64);
//   warps 2..   bf16: read the accumulator once; e4m3: add every K block's sums, scaled, in registers.
// All waits are bounded; a CTA that gives up still takes part in the cluster's barriers.
#pragma once

#include <cuda_bf16.h>

#include <algorithm>
#include <atomic>

#include "fused_select.hpp"
#include "gemm2_core.cuh"
#include "gemm_core.cuh"
#include "gemm_select.hpp"
#include "sm100_ptx.cuh"

namespace rocshmem {
namespace kernels {
namespace gemms {

constexpr int BM = 128;
constexpr int SLAB_BYTES = 128;
constexpr int threads(int bn) { return 64 + 128 * (bn / 64); }   // four epilogue warps for each 64 columns
constexpr int MAX_SPLIT = 8;                         // a portable cluster
constexpr unsigned long long WAIT_BUDGET_NS = gemm::WAIT_BUDGET_NS;

constexpr int MAX_STAGES = 16;
constexpr int MIN_SMEM = 80 * 1024;                  // two CTAs an SM at most: each takes up to half of the TMEM
constexpr int SMEM_LIMIT = 225 * 1024;               // of 227 KiB; the barriers take some of the rest
// Row of the partial tile in shared memory, padded: conflict-free 16-byte accesses with a row per thread.
constexpr int part_row_floats(int bn) { return bn + 4; }

struct Shared {
  uint64_t full[MAX_STAGES];
  uint64_t empty[MAX_STAGES];
  uint64_t tmem_full[2];
  uint64_t tmem_empty[2];
  uint32_t tmem_base;
  volatile int abort_flag;
};

__device__ __forceinline__ float4 ld_cluster_f4(uint32_t cluster_addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(cluster_addr) : "memory");
  return v;
}

struct Args {
  __nv_bfloat16 *c;
  const float *a_scale, *b_scale;   // e4m3 only
  int m, n, k_slabs, tiles_n, split;
  int a_box_rows, stages;           // rows of A that a stage holds (a multiple of eight), stages of the ring
};

template <bool FP8, int BN>
__device__ __forceinline__ void run(const CUtensorMap *map_a, const CUtensorMap *map_b, const Args &a,
                                    unsigned char *smem_raw, Shared &sh) {
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  unsigned char *smem = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  constexpr int PART_ROW_FLOATS = part_row_floats(BN);
  // A stage holds the rows of A that exist and then B. The MMA always reads 128 rows: what follows the stored ones is
  // other shared memory and ends up in result rows that nobody reads.
  const int stages = a.stages, a_bytes = a.a_box_rows * SLAB_BYTES, stage_bytes = a_bytes + BN * SLAB_BYTES;
  constexpr int SLAB_ELEMS = FP8 ? SLAB_BYTES : SLAB_BYTES / 2;
  constexpr int TMEM_COLS = FP8 ? 2 * BN : BN;   // e4m3: two buffers, so that the tensor core runs one K block ahead
  constexpr uint32_t IDESC = sm100::make_idesc(BM, BN, FP8 ? sm100::kFormatE4M3 : sm100::kFormatBF16);
  const int rank = blockIdx.x % a.split, tile = blockIdx.x / a.split;
  const int row0 = tile / a.tiles_n * BM, col0 = tile % a.tiles_n * BN;
  const int rows = min(BM, a.m - row0), cols = min(BN, a.n - col0);
  const int ks0 = static_cast<int>(static_cast<long long>(a.k_slabs) * rank / a.split);
  const int ks1 = static_cast<int>(static_cast<long long>(a.k_slabs) * (rank + 1) / a.split);

  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      sm100::mbar_init(&sh.full[s], 1);
      sm100::mbar_init(&sh.empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      sm100::mbar_init(&sh.tmem_full[b], 1);
      sm100::mbar_init(&sh.tmem_empty[b], BN / 16);
    }
    sh.abort_flag = 0;
    sm100::mbar_fence_init();
    sm100::tma_prefetch_desc(map_a);
    sm100::tma_prefetch_desc(map_b);
  }
  if (warp == 1) sm100::tmem_alloc(&sh.tmem_base, TMEM_COLS);
  sm100::tcgen05_fence_before();
  __syncthreads();
  sm100::tcgen05_fence_after();
  const uint32_t tmem_base = sh.tmem_base;

  if (warp == 0) {
    if (lane == 0) {
      uint32_t stage = 0, phase = 0;
      for (int ks = ks0; ks < ks1; ++ks) {
        if (!sm100::mbar_wait(&sh.empty[stage], phase ^ 1u, &sh.abort_flag, WAIT_BUDGET_NS)) break;
        unsigned char *sa = smem + stage * stage_bytes;
        sm100::mbar_arrive_expect_tx(&sh.full[stage], static_cast<uint32_t>(stage_bytes));
        sm100::tma_load_2d(sa + a_bytes, map_b, &sh.full[stage], ks * SLAB_ELEMS, col0);
        sm100::tma_load_2d(sa, map_a, &sh.full[stage], ks * SLAB_ELEMS, row0);
        if (static_cast<int>(++stage) == stages) { stage = 0; phase ^= 1u; }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      uint32_t stage = 0, phase = 0, buf = 0, buf_phase = 0;
      for (int ks = ks0; ks < ks1; ++ks) {
        if (FP8 && !sm100::mbar_wait(&sh.tmem_empty[buf], buf_phase ^ 1u, &sh.abort_flag, WAIT_BUDGET_NS)) break;
        if (!sm100::mbar_wait(&sh.full[stage], phase, &sh.abort_flag, WAIT_BUDGET_NS)) break;
        sm100::tcgen05_fence_after();
        const uint32_t sa = sm100::smem_u32(smem + stage * stage_bytes);
        const uint64_t da = sm100::make_sw128_desc(sa), db = sm100::make_sw128_desc(sa + a_bytes);
#pragma unroll
        for (int kk = 0; kk < SLAB_BYTES / 32; ++kk) {
          if (FP8) sm100::mma_f8(tmem_base + buf * BN, da + 2 * kk, db + 2 * kk, IDESC, kk != 0);
          else sm100::mma_f16(tmem_base, da + 2 * kk, db + 2 * kk, IDESC, ks != ks0 || kk != 0);
        }
        sm100::mma_commit(&sh.empty[stage]);
        if (FP8) sm100::mma_commit(&sh.tmem_full[buf]);
        if (static_cast<int>(++stage) == stages) { stage = 0; phase ^= 1u; }
        if (FP8) {
          buf ^= 1u;
          if (buf == 0) buf_phase ^= 1u;
        }
      }
      if (!FP8 && !sh.abort_flag) sm100::mma_commit(&sh.tmem_full[0]);
    }
  } else {
    // TMEM lanes [32 * quarter, +32) belong to this warp; it takes 64 of the tile's columns.
    const int quarter = warp & 3, row = quarter * 32 + lane, first_col = (warp - 2) / 4 * 64;
    const uint32_t tlane = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + first_col;
    float *part = reinterpret_cast<float *>(smem) + row * PART_ROW_FLOATS + first_col;
    if constexpr (FP8) {
      const float *sa = a.a_scale + static_cast<size_t>(row0 + (row < rows ? row : 0)) * a.k_slabs;
      const float *sb = a.b_scale + static_cast<size_t>(col0 / 128) * a.k_slabs;
      unsigned long long acc[32];
#pragma unroll
      for (int i = 0; i < 32; ++i) acc[i] = 0ull;
      uint32_t buf = 0, buf_phase = 0;
      float next[4];   // the scales of four K blocks, fetched while the four before them are added
#pragma unroll
      for (int j = 0; j < 4; ++j) next[j] = ks0 + j < ks1 ? sa[ks0 + j] * sb[ks0 + j] : 0.f;
      for (int ks = ks0; ks < ks1 && !sh.abort_flag; ks += 4) {
        float cur[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          cur[j] = next[j];
          next[j] = ks + 4 + j < ks1 ? sa[ks + 4 + j] * sb[ks + 4 + j] : 0.f;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (ks + j >= ks1) break;
          if (!sm100::mbar_wait(&sh.tmem_full[buf], buf_phase, &sh.abort_flag, WAIT_BUDGET_NS)) break;
          sm100::tcgen05_fence_after();
          const unsigned long long s2 = sm100::pack_f32x2(cur[j], cur[j]);
          const uint32_t taddr = tlane + buf * BN;
          uint32_t v[64];
          sm100::tmem_ld_32x64(taddr, v);
          sm100::tmem_ld_wait_for(v);
          sm100::tcgen05_fence_before();   // everything has arrived: the buffer may be overwritten
          __syncwarp();
          if (lane == 0) sm100::mbar_arrive(&sh.tmem_empty[buf]);
          sm100::add_scaled(acc, v, s2);
          buf ^= 1u;
          if (buf == 0) buf_phase ^= 1u;
        }
      }
      // The last K block's sums are here, so all MMAs of this CTA have completed and the ring may be written over.
      if (row < rows) {
#pragma unroll
        for (int q = 0; q < 16; ++q) {
          *reinterpret_cast<float4 *>(part + 4 * q) =
              make_float4(sm100::half_of_f32x2(acc[2 * q], 0), sm100::half_of_f32x2(acc[2 * q], 1),
                          sm100::half_of_f32x2(acc[2 * q + 1], 0), sm100::half_of_f32x2(acc[2 * q + 1], 1));
        }
      }
    } else {
      if (sm100::mbar_wait(&sh.tmem_full[0], 0, &sh.abort_flag, WAIT_BUDGET_NS)) {
        sm100::tcgen05_fence_after();
        uint32_t v[64];
        sm100::tmem_ld_32x64(tlane, v);
        sm100::tmem_ld_wait_for(v);
        if (row < rows) {
#pragma unroll
          for (int q = 0; q < 16; ++q) {
            *reinterpret_cast<uint4 *>(part + 4 * q) = make_uint4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
          }
        }
      }
    }
  }
  __syncwarp();
  if (sh.abort_flag) {
    // Give bulk copies that are still in flight time to land before the shared memory is released.
    unsigned long long t0;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t0));
    for (int i = 0; i < 4096; ++i) {
      unsigned long long now;
      asm volatile("mov.u64 %0, %globaltimer;" : "=l"(now));
      if (now - t0 > 200000ull) break;
      __nanosleep(200);
    }
  }
  sm100::tcgen05_fence_before();
  __syncthreads();
  if (warp == 1) {
    sm100::tcgen05_fence_after();
    sm100::tmem_dealloc(tmem_base, TMEM_COLS);
  }
  // Every CTA's partial tile is in place; eight columns of a row are one unit, unit u belongs to CTA u / threads(BN) % S.
  gemm2::cluster_sync();
  if (!sh.abort_flag) {
    const uint32_t base = sm100::smem_u32(smem);
    for (int u = rank * threads(BN) + threadIdx.x; u < rows * (BN / 8); u += a.split * threads(BN)) {
      const int row = u / (BN / 8), col = u % (BN / 8) * 8;
      if (col >= cols) continue;
      const uint32_t off = base + static_cast<uint32_t>((row * PART_ROW_FLOATS + col) * 4);
      float f[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) f[i] = 0.f;
#pragma unroll
      for (int s = 0; s < MAX_SPLIT; ++s) {
        if (s < a.split) {
          const uint32_t from = gemm2::mapa(off, static_cast<uint32_t>(s));
          const float4 lo = ld_cluster_f4(from), hi = ld_cluster_f4(from + 16);
          f[0] += lo.x; f[1] += lo.y; f[2] += lo.z; f[3] += lo.w;
          f[4] += hi.x; f[5] += hi.y; f[6] += hi.z; f[7] += hi.w;
        }
      }
      __nv_bfloat16 *dst = a.c + static_cast<size_t>(row0 + row) * a.n + col0 + col;
      int4 packed;
      __nv_bfloat162 *p = reinterpret_cast<__nv_bfloat162 *>(&packed);
#pragma unroll
      for (int i = 0; i < 4; ++i) p[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
      if (col + 8 <= cols && (reinterpret_cast<uintptr_t>(dst) & 15u) == 0) {
        *reinterpret_cast<int4 *>(dst) = packed;
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          if (col + i < cols) dst[i] = i & 1 ? p[i / 2].y : p[i / 2].x;
        }
      }
    }
  }
  // Nobody leaves while a neighbour may still read its partial tile.
  __syncwarp();
  gemm2::cluster_sync();
  if (threadIdx.x == 0 && sh.abort_flag) atomicAdd(&gemm::g_gemm_errors, 1u);
}

template <auto Kernel>
inline cudaError_t allow_smem() {
  return cudaFuncSetAttribute(Kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_LIMIT);
}

// How many clusters of `split` CTAs the GPU runs at once (a cluster stays inside a GPC, so 15 of eight and 33 of four
// on 148 SMs), asked until it is answered, once for each size. 0: not at all.
template <auto Kernel>
inline int clusters_at_once(int split, int bn) {
  static std::atomic<int> known[MAX_SPLIT + 1] = {};   // answer + 1; 0: none yet. Every thread would find the same.
  const int n = known[split].load(std::memory_order_relaxed);
  if (n == 0) {
    if (allow_smem<Kernel>() != cudaSuccess) {
      cudaGetLastError();
      return 0;
    }
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = static_cast<unsigned>(split);
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(static_cast<unsigned>(split));
    cfg.blockDim = dim3(threads(bn));
    cfg.dynamicSmemBytes = SMEM_LIMIT;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int found = 0;
    if (cudaOccupancyMaxActiveClusters(&found, Kernel, &cfg) != cudaSuccess) {
      cudaGetLastError();
      return 0;
    }
    known[split].store(found + 1, std::memory_order_relaxed);
    return found;
  }
  return n - 1;
}
// CTAs that share each of `tiles` tiles: as many as run at once, each with at least four K slabs. 0: more tiles than the
// GPU takes at once, or fewer CTAs a tile than `least`: the persistent kernels with their larger tiles are better.
template <auto Kernel>
inline int split_for(long long tiles, int k_slabs, int bn, int least) {
  for (int s = MAX_SPLIT; s > 1 && s >= least; s /= 2) {
    if (k_slabs >= 4 * s && tiles <= clusters_at_once<Kernel>(s, bn)) return s;
  }
  return least <= 1 && tiles <= clusters_at_once<Kernel>(1, bn) ? 1 : 0;
}

// Runs the product if it has few enough tiles and its result shares no memory with an operand (the persistent kernels
// compute up to 128 x 256 or 256 x 256 results in one piece, which reads all of A and B before it writes; here a
// neighbouring tile may still be reading); returns -2 if not, else 0, a cudaError_t, or -1 when the driver cannot
// encode tensor maps. `least`: see split_least_bf16; 2 for e4m3, where a tile of half the width costs the accumulate warps
// more than half the time (96 to 144 tiles of one CTA against the persistent kernel's half as many, 256 to 2048 rows:
// 5 - 19 % slower in all 36 shapes with a K of 512 to 4096, e.g. 512 x 4096 x 4096 24.7 us against 20.6, and within 3 %
// at 7168). `Wide` and `Narrow` are run<FP8, 128> and run<FP8, 64> behind __launch_bounds__(threads(BN), 1);
// narrow tiles are taken where they keep more CTAs busy (64 x 2048: 16 wide tiles x 4 CTAs, 32 narrow ones x 4).
// `encode(map, base, rows, box_rows)` makes the K-slab map of an operand.
template <auto Wide, auto Narrow, typename Encode>
inline int try_launch(const void *a, const void *b, void *c, const float *a_scale,
                      const float *b_scale, int m, int n, int k_bytes, int least, Encode encode, cudaStream_t stream) {
  const Span result{c, size_t(m) * n * 2};
  if (overlaps(result, Span{a, size_t(m) * k_bytes}) || overlaps(result, Span{b, size_t(n) * k_bytes})) return -2;
  Args args{static_cast<__nv_bfloat16 *>(c), a_scale, b_scale, m, n, (k_bytes + SLAB_BYTES - 1) / SLAB_BYTES, 0, 0,
            m < BM ? (m + 7) / 8 * 8 : BM, 0};
  const long long row_blocks = (m + BM - 1) / BM, wide_tiles = row_blocks * ((n + 127) / 128),
                  narrow_tiles = row_blocks * ((n + 63) / 64);
  const int ws = split_for<Wide>(wide_tiles, args.k_slabs, 128, least);
  const int ns = split_for<Narrow>(narrow_tiles, args.k_slabs, 64, least);
  if (ws == 0 && ns == 0) return -2;
  const bool take_narrow = narrow_tiles * ns > wide_tiles * ws;
  const int bn = take_narrow ? 64 : 128;
  args.tiles_n = (n + bn - 1) / bn;
  args.split = take_narrow ? ns : ws;
  // The ring takes what shared memory is left: a decode step is bound by the bytes in flight (32 x 7168 x 8192 bf16: eleven
  // stages of 20 KiB). Behind it lies what an MMA reads past a short last stage (128 rows of A), in front the alignment.
  const int stage_bytes = (args.a_box_rows + bn) * SLAB_BYTES;
  const int overrun = std::max(0, BM * SLAB_BYTES - stage_bytes);
  const int slabs_each = (args.k_slabs + args.split - 1) / args.split;
  const int for_part = (std::min(m, BM) * part_row_floats(bn) * 4 + stage_bytes - 1) / stage_bytes;
  args.stages = std::min({(SMEM_LIMIT - 1024 - overrun) / stage_bytes, MAX_STAGES, std::max(slabs_each, for_part)});
  CUtensorMap map_a, map_b;
  if (!encode(&map_a, a, m, args.a_box_rows) || !encode(&map_b, b, n, bn)) return -1;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = static_cast<unsigned>(args.split);
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>(row_blocks * args.tiles_n * args.split));
  cfg.blockDim = dim3(threads(bn));
  cfg.dynamicSmemBytes = static_cast<size_t>(std::max(MIN_SMEM, args.stages * stage_bytes + overrun + 1024));
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const cudaError_t e = take_narrow ? allow_smem<Narrow>() : allow_smem<Wide>();
  if (e != cudaSuccess) return static_cast<int>(e);
  return static_cast<int>(cudaLaunchKernelEx(&cfg, take_narrow ? Narrow : Wide, map_a, map_b, args));
}

}  // namespace gemms
}  // namespace kernels
}  // namespace rocshmem
