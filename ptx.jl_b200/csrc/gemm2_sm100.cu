// gemm_bf16 on CTA pairs: one output tile of 256 rows and 128, 192 or 256 columns per pair of SMs, issued as
// tcgen05.mma.cta_group::2.
//
// Why a second GEMM kernel. The single-CTA kernel (gemm_sm100.cu) streams 48 KiB
// from L2 into shared memory per 128x256x64 block of work; at the tensor pipe's rate
// that is ~17 TB/s over the 148 SMs, and a profile of 8192^3 shows the pipe active
// 82 % of the time with the rest spent waiting for operands. A CTA pair splits one
// 256x256 tile so that each SM holds only ITS 128 rows of A and ITS 128 rows of B^T
// per k-step (32 KiB for the same work: a third less traffic, and a six-deep ring in
// the same shared memory); the pair's leader issues m256n256k16 instructions that
// read both halves, and each SM ends up with its 128 rows of the 256-column
// accumulator in its own tensor memory. The reference has no counterpart (its GEMM is
// cta_group::1 throughout, test/gpu/blackwell/gemm_highperf_blackwell.jl:69-199).
//
// Roles in EACH CTA of the pair (192 threads): warp 0 TMA producer, warp 1 MMA
// (issues only in the leader; in both it owns the tensor-memory allocation), warps 2-5
// epilogue. Barriers live at the same shared-memory offsets in both CTAs:
//   full[s]      leader's only: two arrivals (each CTA's producer posts its own byte
//                count) plus the bytes of both CTAs' TMA loads, which name the leader's
//                barrier (cta_group::2 loads may signal the peer's barrier);
//   empty[s]     own: the leader commits to its own and to the peer's;
//   acc_full[b]  own: likewise two commits by the leader;
//   acc_empty[b] leader's only: 128 epilogue threads of each CTA arrive (remotely from
//                the peer) once their rows of the accumulator are in registers.
// No load is multicast; the peer's barriers are reached through mapa-translated
// addresses. Every wait is bounded as in the single-CTA kernel, and the pair meets at a
// cluster barrier before the first remote arrival and before exit.
//
// Work per launch: 2*G*M*N*K flop; compulsory bytes G*((M*K + N*K)*2 + M*N*sizeof(out)).
#include "cta_pair.cuh"
#include "gemm_epilogue.cuh"
#include "host_common.h"
#include "sm100_prims.cuh"

namespace ptxb200 {
namespace {

constexpr int kBM2 = 256;                      // rows of the pair's tile (128 per CTA)
constexpr int kBK2 = 64;
constexpr int kAStage2 = 128 * kBK2 * 2;       // this CTA's 128 rows of A: 16 KiB
constexpr int kThreads2 = 192;
constexpr int kAccCols2 = 256;                 // distance of the two accumulators in tensor memory
constexpr int kGroupM2 = 8;                    // row-tiles (of 256) per rasterisation band

// kBN columns of the pair's tile: 128, 192 or 256
template <int kBN>
struct Cfg2 {
  static constexpr int kBStage = kBN / 2 * kBK2 * 2;   // this CTA's half of the rows of B^T
  static constexpr int kStage = kAStage2 + kBStage;
  static constexpr int kStages = kBN == 256 ? 6 : kBN == 192 ? 8 : 9;
  static constexpr int kOffA = 0;
  static constexpr int kOffB = kOffA + kStages * kAStage2;
  static constexpr int kOffBars = kOffB + kStages * kBStage;   // full[] empty[] acc_full[2] acc_empty[2]
  static constexpr int kOffTmemSlot = kOffBars + (2 * kStages + 4) * 8;
  static constexpr int kOffAbort = kOffTmemSlot + 8;
  static constexpr int kSmemBytes = kOffAbort + 8;      // the base must be 1024-byte aligned (checked)
  static_assert(kSmemBytes <= 232448, "exceeds the 227 KiB a CTA can opt in to");
};

enum : uint32_t { kSite2Empty = 18, kSite2Full = 19, kSite2AccEmpty = 20, kSite2AccFull = 21 };

__device__ __forceinline__ void tile_coords2(int tile, int tiles_m, int tiles_n, int& tm, int& tn) {
  const int band_tiles = kGroupM2 * tiles_n;
  const int band = tile / band_tiles;
  const int first_m = band * kGroupM2;
  const int rows_in_band = min(tiles_m - first_m, kGroupM2);
  const int r = tile - band * band_tiles;
  tm = first_m + r % rows_in_band;
  tn = r / rows_in_band;
}

template <int kBN, bool kF32Out>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads2, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                 void* __restrict__ c_out, int M, int N, int K, int ldc, int groups, uint32_t* status) {
  using C = Cfg2<kBN>;
  constexpr int kStages2 = C::kStages;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw;
  const uint32_t base = smem_u32(smem_raw);
  const uint32_t rank = cluster_ctarank();        // 0: the pair's leader
  const bool leader = rank == 0;

  const uint32_t a_base = base + C::kOffA;
  const uint32_t b_base = base + C::kOffB;
  const uint32_t bar_full = base + C::kOffBars;
  const uint32_t bar_empty = bar_full + kStages2 * 8;
  const uint32_t bar_acc_full = bar_empty + kStages2 * 8;
  const uint32_t bar_acc_empty = bar_acc_full + 2 * 8;
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem + C::kOffTmemSlot);
  volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(smem + C::kOffAbort);
  const WaitCtx wctx{status, abort_flag};

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  // the swizzled tiles need a 1024-byte aligned base; both CTAs of a pair see the same offset
  const bool misaligned = (base & 1023u) != 0;
  if (misaligned && threadIdx.x == 0 && status != nullptr) {
    grid_wait();
    atomicCAS(status, 0u, kStatusTimeoutTag | (17u << 8));
  }

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int s = 0; s < kStages2; ++s) {
      mbar_init(bar_full + 8 * s, 2);      // one arrival per CTA of the pair (used in the leader)
      mbar_init(bar_empty + 8 * s, 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(bar_acc_full + 8 * b, 1);
      mbar_init(bar_acc_empty + 8 * b, 256);   // 128 epilogue threads per CTA (used in the leader)
    }
    mbar_fence_init();
  }
  if (warp == 1 && !misaligned) {
    tmem_alloc_pair(smem_u32(const_cast<uint32_t*>(tmem_slot)), 512);
    tmem_relinquish_pair();
  }
  grid_wait();
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();     // both CTAs' barriers exist before anything remote is signalled
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  const int tiles_m = (M + kBM2 - 1) / kBM2;   // M % 128 == 0: the last row-tile may be its first half only
  const int tiles_n = (N + kBN - 1) / kBN;
  const int tiles_per_group = tiles_m * tiles_n;
  const int total_tiles = tiles_per_group * groups;
  const int kiters = K / kBK2;
  const int pair = blockIdx.x >> 1;
  const int pairs = gridDim.x >> 1;

  if (misaligned) {
    // nothing was allocated; leave together
  } else if (warp == 0) {
    // ---------------- TMA producer (both CTAs) ----------------
    if (elect_one()) {
      tma_prefetch_desc(&tmap_a);
      tma_prefetch_desc(&tmap_b);
      const uint32_t leader_full = map_to_cta(bar_full, 0);
      uint32_t it = 0;
      for (int tile = pair; tile < total_tiles; tile += pairs) {
        int tm, tn;
        const int g = tile / tiles_per_group;
        tile_coords2(tile - g * tiles_per_group, tiles_m, tiles_n, tm, tn);
        const int a_row = g * M + tm * kBM2 + (int)rank * 128;
        const int b_row = g * N + tn * kBN + (int)rank * (kBN / 2);
        for (int k = 0; k < kiters; ++k, ++it) {
          const uint32_t s = it % kStages2;
          const uint32_t ph = (it / kStages2) & 1u;
          mbar_wait(bar_empty + 8 * s, ph ^ 1u, wctx, kSite2Empty);
          mbar_arrive_expect_tx_cluster(leader_full + 8 * s, C::kStage);
          tma_load_2d_pair(a_base + s * kAStage2, &tmap_a, k * kBK2, a_row, leader_full + 8 * s);
          tma_load_2d_pair(b_base + s * C::kBStage, &tmap_b, k * kBK2, b_row, leader_full + 8 * s);
        }
      }
      grid_trigger();
    }
  } else if (warp == 1) {
    // ---------------- MMA issue (leader only; converged warp, elected lane) ----------------
    if (leader) {
      constexpr uint32_t idesc = make_idesc_bf16_f32(kBM2, kBN, false, false);
      const uint32_t peer_empty = map_to_cta(bar_empty, 1);
      const uint32_t peer_acc_full = map_to_cta(bar_acc_full, 1);
      uint32_t it = 0, t = 0;
      for (int tile = pair; tile < total_tiles; tile += pairs, ++t) {
        const uint32_t buf = t & 1u;
        const uint32_t aph = (t >> 1) & 1u;
        mbar_wait_warp(bar_acc_empty + 8 * buf, aph ^ 1u, wctx, kSite2AccEmpty);
        tc_fence_after();
        const uint32_t d_tmem = tmem + buf * kAccCols2;
        for (int k = 0; k < kiters; ++k, ++it) {
          const uint32_t s = it % kStages2;
          const uint32_t ph = (it / kStages2) & 1u;
          mbar_wait_warp(bar_full + 8 * s, ph, wctx, kSite2Full);
          tc_fence_after();
          const uint32_t da = sdesc_lo(a_base + s * kAStage2, 16);
          const uint32_t db = sdesc_lo(b_base + s * C::kBStage, 16);
          constexpr uint32_t dhi = sdesc_hi(1024, kLayoutB128);
#pragma unroll
          for (int kk = 0; kk < kBK2 / 16; ++kk)
            tc_mma_ss_pair(d_tmem, da + 2 * kk, dhi, db + 2 * kk, dhi, idesc, (k | kk) != 0 ? 1u : 0u);
          tc_commit_pair(bar_empty + 8 * s);      // this CTA's slot
          tc_commit_pair(peer_empty + 8 * s);     // the peer's slot
        }
        tc_commit_pair(bar_acc_full + 8 * buf);
        tc_commit_pair(peer_acc_full + 8 * buf);
      }
    }
  } else {
    // ---------------- epilogue (both CTAs): this CTA's 128 rows of the tile ----------------
    const int quad = warp & 3;
    const uint32_t leader_acc_empty = map_to_cta(bar_acc_empty, 0);
    uint32_t t = 0;
    for (int tile = pair; tile < total_tiles; tile += pairs, ++t) {
      int tm, tn;
      const int g = tile / tiles_per_group;
      tile_coords2(tile - g * tiles_per_group, tiles_m, tiles_n, tm, tn);
      const uint32_t buf = t & 1u;
      const uint32_t aph = (t >> 1) & 1u;
      mbar_wait(bar_acc_full + 8 * buf, aph, wctx, kSite2AccFull);
      tc_fence_after();
      // in a half-filled last row-tile the peer's 128 rows lie past M (its A box read the
      // next group's rows or zero fill): computed, not stored
      const bool rows_valid = tm * kBM2 + (int)rank * 128 < M;
      const int col0 = tn * kBN;
#pragma unroll 1
      for (int h = 0; h < 2; ++h) {          // this warp's first and second 16 rows
        const size_t row = (size_t)g * M + (size_t)tm * kBM2 + rank * 128 + quad * 32 + h * 16 + (lane >> 2);
        const uint32_t t_row = tmem_addr(tmem, quad * 32 + h * 16, buf * kAccCols2);
#pragma unroll 1
        for (int c = 0; c < kBN; c += 64) {
          uint32_t v[32];
          tmem_ld_16x64(t_row + c, v);
          tc_wait_ld_bind(v);
          if (col0 + c < N && rows_valid) store_acc_16x64<kF32Out>(c_out, row, ldc, col0 + c, v);   // N % 64 == 0
        }
      }
      tc_fence_before();
      mbar_arrive_cluster(leader_acc_empty + 8 * buf);
    }
  }

  // Neither CTA may leave (or free tensor memory) while the other can still signal
  // its barriers or while the leader's instructions still read its shared memory.
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  if (warp == 1 && !misaligned) {
    tc_fence_after();
    tmem_dealloc_pair(tmem, 512);
  }
}

}  // namespace

// Columns of the pair's tile for a product, or 0 where 128x256 tiles of single CTAs
// (gemm_sm100.cu) are the better choice. The estimate, in us: rounds over the machine times
// what a tile costs, which is its steps of K (0.345, 0.27, 0.215 us for 256, 192, 128 columns;
// single CTAs 0.36) or, for short K, its epilogue (0.3 us + 0.004 per column), plus one epilogue.
// Wide tiles cost least per column; narrower ones are taken where they fill the last round
// better: 2304x2304x1024 16.2 us with 256 columns, 13.9 with 192; 1792x1792x8192 43.7 and
// 36.8; 48 products of 256x320x512 13.1 with 256, 11.4 with 128; the other way round
// 8192x8192x512 50.9 with 256, 65.9 with 128 and 8192^3 694 and 833. Single CTAs win where M leaves half
// of a pair's last row-tile empty (32 products of 128x2048x2048: 59.3 us in pairs, 52.8
// single). Any width gives the same bits: an element is one accumulation in k order.
int gemm_pair_tile(const DeviceCtx& ctx, int groups, int M, int N, int K) {
  const double kiters = K / kBK2;
  auto cost = [&](long long tiles, long long at_once, double step, int bn) {
    const double epilogue = 0.3 + 0.004 * bn, tile = kiters * step > epilogue ? kiters * step : epilogue;
    return (double)((tiles + at_once - 1) / at_once) * tile + epilogue;
  };
  const int pairs = ctx.sm_count / 2;
  const long long row_tiles = (long long)groups * ((M + kBM2 - 1) / kBM2);   // a last row-tile may be half-filled
  int best = 0;
  double least = cost((long long)groups * (M / 128) * ((N + 255) / 256), ctx.sm_count, 0.36, 256) + 1.0;
  const int bns[3] = {256, 192, 128};
  const double steps[3] = {0.345, 0.27, 0.215};
  for (int i = 0; i < 3; ++i) {
    const double c = cost(row_tiles * ((N + bns[i] - 1) / bns[i]), pairs, steps[i], bns[i]);
    if (c < least) {
      least = c;
      best = bns[i];
    }
  }
  return best;
}

namespace {

template <int kBN, bool kF32Out>
int launch_one2(const DeviceCtx& ctx, void* C, const void* A, const void* Bt, int groups, int M, int N, int K, int ldc,
                cudaStream_t stream) {
  CUtensorMap ta, tb;
  int rc = encode_tmap_bf16_2d(&ta, A, (uint64_t)groups * M, (uint64_t)K, (uint64_t)K * 2, 128, kBK2);
  if (rc != PTXB200_OK) return rc;
  rc = encode_tmap_bf16_2d(&tb, Bt, (uint64_t)groups * N, (uint64_t)K, (uint64_t)K * 2, kBN / 2, kBK2);
  if (rc != PTXB200_OK) return rc;
  static PerDeviceOnce attr_once;
  rc = attr_once.run(ctx.device, []() -> int {
    PTXB200_CUDA_TRY(cudaFuncSetAttribute(gemm_pair_kernel<kBN, kF32Out>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          Cfg2<kBN>::kSmemBytes));
    return PTXB200_OK;
  });
  if (rc != PTXB200_OK) return rc;
  const long long tiles = (long long)groups * ((M + kBM2 - 1) / kBM2) * ((N + kBN - 1) / kBN);
  const int max_pairs = ctx.sm_count / 2;
  const int pairs = tiles < max_pairs ? (int)tiles : max_pairs;
  // (the cluster's size is the kernel's own)
  PTXB200_CUDA_TRY(launch_after(stream, gemm_pair_kernel<kBN, kF32Out>, 2u * pairs, kThreads2, Cfg2<kBN>::kSmemBytes, 1u, ta, tb, C,
                                M, N, K, ldc, groups, status_word(ctx, stream)));
  return PTXB200_OK;
}

}  // namespace

int launch_gemm_pair(const DeviceCtx& ctx, int bn, void* C, const void* A, const void* Bt, int groups, int M, int N,
                     int K, int ldc, unsigned flags, cudaStream_t stream) {
  const bool f32 = (flags & PTXB200_GEMM_F32_OUT) != 0;
#define PTXB200_PAIR_TILE(BN)                                                                           \
  if (bn == BN)                                                                                         \
    return f32 ? launch_one2<BN, true>(ctx, C, A, Bt, groups, M, N, K, ldc, stream)                     \
               : launch_one2<BN, false>(ctx, C, A, Bt, groups, M, N, K, ldc, stream)
  PTXB200_PAIR_TILE(128);
  PTXB200_PAIR_TILE(192);
  PTXB200_PAIR_TILE(256);
#undef PTXB200_PAIR_TILE
  return PTXB200_E_INVALID;
}

}  // namespace ptxb200
