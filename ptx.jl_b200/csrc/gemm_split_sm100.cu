// gemm_bf16 for products with too few large tiles to fill the machine: one 128-row tile of
// 64, 128 or 192 columns per CTA, with K split over the 1 to 8 CTAs of a cluster.
//
// What bounds such a product is not the tensor pipe but one CTA's chain: launch, tensor
// maps, first loads, then about 0.16 us (64 columns), 0.19 (128) or 0.25 (192) per step of 64
// of K -- shared memory takes in and feeds out 24, 32 or 40 KiB per step -- and the epilogue. So the
// work is spread over as many CTAs as there are SMs: small tiles first, then K. The parts
// of a tile meet inside the cluster: every CTA sends each other one its share of the
// columns of the partial sums with asynchronous stores into that CTA's shared memory
// (counted on an mbarrier there), adds up its own share in the order of the parts, and
// writes it. Nothing goes through global memory, there is no second kernel, and no CTA
// waits for one that the hardware has not co-scheduled with it. The order of the sums is
// fixed, so results are reproducible (they differ in the last bits from the unsplit order).
// One-shot blocks: the first loads are issued before the block's threads even meet.
//
// A CTA sums its part of K in several chains: the tensor core's fp32 accumulation loses about
// 5e-8 of the result per step of a chain (1024x1152x8192 split in 2, fp32 out: one chain of 64
// steps 4.0e-6, four of 16 8.5e-7, of 8 4.0e-7). With fp32 output a chain has at most 8 steps where
// the accumulators suffice (64 columns: 8 of them, 128: 4), and with either output never more
// than the shares of one line of steps over all SMs would (gemm_line: 8 to 62). Where K is split
// each chain has an accumulator of its own and the epilogue adds them up; with more chains than
// that two accumulators take turns and the epilogue's warps fold them into a third as they end,
// which costs 0.1 us per chain (128x256x65536 in 4 parts, fp32 out: 32 chains 48.5 us and 4.1e-7, 8
// chains of 32 steps 47.4 and 1.9e-6; in 8 parts 39.6 and 4.0e-7). Where K is not split the
// epilogue's warps take each chain into registers while the next one runs (1024x1280x4096: fp32
// out 18.6 us in chains of 8, bf16 17.8 in chains of 16, 17.0 in one).
//
// Measured (device time, bf16 out unless noted; before: 128x256 tiles cut into shares of
// one k-iteration line, partial tiles parked in global memory, a second kernel to add
// them up): 128x4096x4096 19.1 -> 12.5 us; 1024x1152x8192 fp32 out 33.1 -> 23.0; 1024^3
// 14.5 -> 6.6; 512^3 8.0 -> 4.9; 128x128x8192 14.9 -> 9.7; 128x256x65536 61.0 -> 39.3.
//
// Algorithmic work per launch: 2*G*M*N*K flop; compulsory bytes G*((M*K + N*K)*2 +
// M*N*sizeof(out)).
#include "cta_pair.cuh"
#include "gemm_epilogue.cuh"
#include "host_common.h"

namespace ptxb200 {
namespace {

constexpr int kThreads3 = 192;        // warp 0 TMA producer, warp 1 MMA, warps 2-5 epilogue
constexpr int kBandM3 = 8;            // row-tiles per rasterisation band

enum : uint32_t { kSite3Empty = 24, kSite3Full = 25, kSite3AccFull = 26, kSite3Parts = 27, kSite3AccEmpty = 28 };

// 16 columns of this thread's row, summed over `pieces` blocks of kBN columns
template <int kBN>
__device__ __forceinline__ void load_sum16(uint32_t taddr, int pieces, float (&x)[16]) {
  uint32_t v[16];
  tmem_ld16(taddr, v);
  tc_wait_ld_bind16(v);
#pragma unroll
  for (int i = 0; i < 16; ++i) x[i] = __uint_as_float(v[i]);
#pragma unroll 1
  for (int a = 1; a < pieces; ++a) {
    tmem_ld16(taddr + a * kBN, v);
    tc_wait_ld_bind16(v);
#pragma unroll
    for (int i = 0; i < 16; ++i) x[i] += __uint_as_float(v[i]);
  }
}

// Adds a finished chain (kBN columns at `acc`) to the columns at `run`, or copies it there.
template <int kBN>
__device__ __forceinline__ void fold_chain(uint32_t run, uint32_t acc, bool copy) {
#pragma unroll 1
  for (int c = 0; c < kBN; c += 32) {
    uint32_t v[32];
    tmem_ld32(acc + c, v);
    tc_wait_ld_bind(v);
    if (!copy) {
      uint32_t x[32];
      tmem_ld32(run + c, x);
      tc_wait_ld_bind(x);
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] = __float_as_uint(__uint_as_float(x[i]) + __uint_as_float(v[i]));
    }
    tmem_st32(run + c, v);
  }
  tc_wait_st();
}

// Adds a finished chain (kBN columns at t_row) to this thread's sums, or takes it as they are: the
// fragments of 16 rows x 64 columns that store_acc_16x64 writes, of the warp's first and second
// 16 rows in turn.
template <int kBN>
__device__ __forceinline__ void take_chain(uint32_t t_row, bool copy, float (&sum)[kBN]) {
#pragma unroll
  for (int b = 0; b < kBN / 32; ++b) {
    uint32_t v[32];
    tmem_ld_16x64(t_row + ((uint32_t)(b & 1) << 20) + (b >> 1) * 64, v);
    tc_wait_ld_bind(v);
#pragma unroll
    for (int i = 0; i < 32; ++i)
      sum[b * 32 + i] = copy ? __uint_as_float(v[i]) : sum[b * 32 + i] + __uint_as_float(v[i]);
  }
}

// kSplit: K is split over the CTAs of a cluster; kFold: into more chains than accumulators.
template <int kBN, bool kF32Out, bool kSplit, bool kFold>
__global__ void __launch_bounds__(kThreads3, 1)
gemm_split_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                  void* __restrict__ c_out, int M, int N, int K, int ldc, int split, int stages, int chain_stages,
                  uint32_t tmem_cols, unsigned long long part_cols, int slot_bytes, uint32_t* status) {
  if constexpr (!kSplit) split = 1;
  constexpr int kStageK = stage_k3(kBN), kStageBytes = stage_bytes3(kBN);
  constexpr int kAtomBytes = kABytes3 + kBN * kBK3 * 2;
  extern __shared__ __align__(1024) uint8_t smem[];
  const uint32_t base = smem_u32(smem);
  const int part = kSplit ? (int)cluster_ctarank() : 0;   // which part of K this CTA of the cluster sums
  const int my_col = unpack_col3(part_cols, part), my_cols = unpack_col3(part_cols, part + 1) - my_col;   // what it adds up

  const uint32_t ctrl = base + stages * kStageBytes;
  uint8_t* ctrl_ptr = smem + stages * kStageBytes;
  const uint32_t bar_full = ctrl, bar_empty = ctrl + 8 * kMaxStages3, bar_acc_full = ctrl + 16 * kMaxStages3;
  const uint32_t bar_acc_empty = bar_acc_full + 16, bar_parts = bar_acc_empty + 16;
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(ctrl_ptr + 16 * kMaxStages3 + 40);
  volatile uint32_t* abort_flag = tmem_slot + 1;
  const uint32_t recv = ctrl + kCtrlBytes3;
  const float4* recv_ptr = reinterpret_cast<const float4*>(ctrl_ptr + kCtrlBytes3);
  const WaitCtx wctx{status, abort_flag};

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const bool misaligned = (base & 1023u) != 0;   // the swizzled tiles need a 1024-byte aligned base
  if (misaligned && threadIdx.x == 0 && status != nullptr) {
    grid_wait();
    atomicCAS(status, 0u, kStatusTimeoutTag | (17u << 8));
  }

  const int tiles_m = M / kBM3, tiles_n = (N + kBN - 1) / kBN;
  const int tiles_per_group = tiles_m * tiles_n;
  const int tile = blockIdx.x / split;
  const int g = tile / tiles_per_group;
  int tm, tn;
  {
    const int r = tile - g * tiles_per_group;
    const int band = r / (kBandM3 * tiles_n), first = band * kBandM3;
    const int rows = min(tiles_m - first, kBandM3), q = r - band * kBandM3 * tiles_n;
    tm = first + q % rows;
    tn = q / rows;
  }
  const int kiters = K / kBK3;
  const int k0 = part_begin3(kiters, split, part), k1 = part_begin3(kiters, split, part + 1);
  const int steps = (k1 - k0 + kStageK - 1) / kStageK;       // ring stages this CTA fills; the last may be a half
  // Chains of sums over chain_stages each. K split: every one in an accumulator of its own, or
  // (kFold) in the second and the third in turn and added to what the first holds as they end;
  // otherwise in two accumulators in turn, and taken into registers as they end.
  const int chains = (steps + chain_stages - 1) / chain_stages;

  auto load = [&](int i, int s) {
    const uint32_t full = bar_full + 8 * s, dst = base + s * kStageBytes;
    const int k = k0 + i * kStageK, n = kStageK == 1 ? 1 : min(kStageK, k1 - k);
    mbar_arrive_expect_tx(full, n * kAtomBytes);
#pragma unroll
    for (int a = 0; a < kStageK; ++a) {
      if (a >= n) break;
      tma_load_2d(dst + a * kAtomBytes, &tmap_a, (k + a) * kBK3, g * M + tm * kBM3, full);
      tma_load_2d(dst + a * kAtomBytes + kABytes3, &tmap_b, (k + a) * kBK3, g * N + tn * kBN, full);
    }
  };
  // the first loads are under way before the block meets
  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmap_a);
    tma_prefetch_desc(&tmap_b);
    *abort_flag = 0;
    for (int s = 0; s < stages; ++s) {
      mbar_init(bar_full + 8 * s, 1);
      mbar_init(bar_empty + 8 * s, 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(bar_acc_full + 8 * i, 1);
      mbar_init(bar_acc_empty + 8 * i, 128);
    }
    mbar_init(bar_parts, 1);
    mbar_fence_init();
    if (kSplit) mbar_arrive_expect_tx(bar_parts, (split - 1) * kBM3 * 4 * my_cols);
    grid_wait();
    if (!misaligned)
      for (int i = 0; i < stages && i < steps; ++i) load(i, i);
  }
  if (warp == 1 && !misaligned) {
    tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_slot)), tmem_cols);
    tmem_relinquish();
  }
  __syncwarp();
  grid_wait();
  tc_fence_before();
  __syncthreads();
  if (kSplit) cluster_arrive();          // "this CTA has started": waited for ahead of the first store to a peer
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (!misaligned && warp == 0) {
    if (lane == 0) {
      int s = 0;
      uint32_t ph = 0;
      for (int i = stages; i < steps; ++i) {
        mbar_wait(bar_empty + 8 * s, ph, wctx, kSite3Empty);
        load(i, s);
        if (++s == stages) { s = 0; ph ^= 1u; }
      }
      grid_trigger();
    }
    __syncwarp();
  } else if (!misaligned && warp == 1) {
    constexpr uint32_t idesc = make_idesc_bf16_f32(kBM3, kBN, false, false);
    constexpr uint32_t dhi = sdesc_hi(1024, kLayoutB128);
    int s = 0;
    uint32_t ph = 0, acc = tmem, first = 0;     // the chain's accumulator; 0: its first product overwrites it
    auto mma = [&](int a, int slot) {           // one step of K: 4 instructions of 16
      const uint32_t da = sdesc_lo(base + slot * kStageBytes + a * kAtomBytes, 16);
      const uint32_t db = sdesc_lo(base + slot * kStageBytes + a * kAtomBytes + kABytes3, 16);
#pragma unroll
      for (int kk = 0; kk < kBK3 / 16; ++kk)   // 2 descriptor units = 32 bytes = 16 elements of K
        tc_mma_ss_warp(acc, da + 2 * kk, dhi, db + 2 * kk, dhi, idesc, a == 0 && kk == 0 ? first : 1u);
    };
    auto full_stage = [&]() {
      mbar_wait_warp(bar_full + 8 * s, ph, wctx, kSite3Full);
      tc_fence_after();
      mma(0, s);
      if constexpr (kStageK == 2) mma(1, s);
      tc_commit_warp(bar_empty + 8 * s);
      if (++s == stages) { s = 0; ph ^= 1u; }
    };
    auto half_stage = [&]() {
      mbar_wait_warp(bar_full + 8 * s, ph, wctx, kSite3Full);
      tc_fence_after();
      mma(0, s);
    };
    // full stages first, without a branch around any instruction (one in this loop costs
    // about a hundred cycles a step), then a last half stage
    const int full_steps = (k1 - k0) / kStageK;
    if constexpr (kSplit && !kFold) {
      int left = chain_stages;                  // stages until the next chain begins
      for (int i = 0; i < full_steps; ++i) {
        full_stage();
        const bool next = --left == 0;
        first = next ? 0u : 1u;
        acc += next ? (uint32_t)kBN : 0u;
        left = next ? chain_stages : left;
      }
      if (full_steps < steps) half_stage();
      tc_commit_warp(bar_acc_full);
    } else {
      int i = 0;
      for (int c = 0; c < chains; ++c) {
        const int buf = c & 1, end = min(i + chain_stages, steps), full_end = min(end, full_steps);
        if (c >= 2) {
          mbar_wait_warp(bar_acc_empty + 8 * buf, (uint32_t)(c / 2 - 1) & 1u, wctx, kSite3AccEmpty);
          tc_fence_after();
        }
        acc = tmem + (buf + (kFold ? 1 : 0)) * kBN;
        first = 0;
        for (; i < full_end; ++i) {
          full_stage();
          first = 1u;
        }
        if (i < end) {
          half_stage();
          ++i;
        }
        tc_commit_warp(bar_acc_full + 8 * buf);
      }
    }
  }

  const int quad = warp & 3;
  const int row_in_tile = quad * 32 + lane;
  const bool epilogue = warp >= 2 && !misaligned;
  const uint32_t t_row = tmem_addr(tmem, quad * 32, 0);
  const size_t row = (size_t)g * M + (size_t)tm * kBM3 + row_in_tile;
  const int col0 = tn * kBN;
  // f(chain's accumulator, number) as the chains end, beside the products of the next
  auto each_chain = [&](auto f) {
#pragma unroll 1
    for (int c = 0; c < chains; ++c) {
      mbar_wait(bar_acc_full + 8 * (c & 1), (uint32_t)(c / 2) & 1u, wctx, kSite3AccFull);
      tc_fence_after();
      f(t_row + ((c & 1) + (kFold ? 1 : 0)) * kBN, c);
      tc_fence_before();
      mbar_arrive(bar_acc_empty + 8 * (c & 1));
    }
  };
  if constexpr (!kSplit) {
    if (epilogue) {
      float sum[kBN];
      each_chain([&](uint32_t acc, int c) { take_chain<kBN>(acc, c == 0, sum); });
#pragma unroll
      for (int b = 0; b < kBN / 32; ++b) {
        const size_t row16 = (size_t)g * M + (size_t)tm * kBM3 + quad * 32 + (b & 1) * 16 + (lane >> 2);
        const int c = (b >> 1) * 64;
        uint32_t v[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] = __float_as_uint(sum[b * 32 + i]);
        if (col0 + c < N) store_acc_16x64<kF32Out>(c_out, row16, ldc, col0 + c, v);   // N % 64 == 0
      }
    }
  } else {
    if (epilogue) {
      if constexpr (kFold) {
        each_chain([&](uint32_t acc, int c) { fold_chain<kBN>(t_row, acc, c == 0); });
      } else {
        mbar_wait(bar_acc_full, 0, wctx, kSite3AccFull);
        tc_fence_after();
      }
    }
    const int pieces = kFold ? 1 : chains;   // blocks of columns to add up
    // every part sums up and writes its share of the columns: it sends the others theirs
    cluster_wait();
    if (epilogue) {
#pragma unroll 1
      for (int i = 1; i < split; ++i) {
        const int q = part + i < split ? part + i : part + i - split;
        const uint32_t slot = part < q ? part : part - 1;
        const uint32_t dst = map_to_cta(recv + slot * slot_bytes, q) + row_in_tile * 16;
        const uint32_t dst_bar = map_to_cta(bar_parts, q);
        const int first = unpack_col3(part_cols, q), cols = unpack_col3(part_cols, q + 1) - first;
#pragma unroll 2
        for (int c = 0; c < cols; c += 16) {
          float x[16];
          load_sum16<kBN>(t_row + first + c, pieces, x);
#pragma unroll
          for (int j = 0; j < 4; ++j)
            st_async_v4(dst + (c / 4 + j) * (kBM3 * 16), dst_bar, x[4 * j], x[4 * j + 1], x[4 * j + 2], x[4 * j + 3]);
        }
      }
    }
    if (epilogue) {
      if (pieces > 1) {
        // this CTA's own share is added up while the others' is on its way
#pragma unroll 1
        for (int c = 0; c < my_cols; c += 16) {
          float x[16];
          load_sum16<kBN>(t_row + my_col + c, pieces, x);
          uint32_t v[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) v[i] = __float_as_uint(x[i]);
          tmem_st16(t_row + my_col + c, v);
        }
        tc_wait_st();
      }
      mbar_wait<true>(bar_parts, 0, wctx, kSite3Parts);   // other CTAs' stores are read behind it
#pragma unroll 1
      for (int c = 0; c < my_cols; c += 16) {
        float own[16], sum[16];
        load_sum16<kBN>(t_row + my_col + c, 1, own);
#pragma unroll
        for (int i = 0; i < 16; ++i) sum[i] = 0.0f;
        // in the order of the parts, whoever adds them up
#pragma unroll 1
        for (int q = 0; q < split; ++q) {
          const float4* src = recv_ptr + (q < part ? q : q - 1) * (slot_bytes / 16) + (c / 4) * kBM3 + row_in_tile;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            float4 x = make_float4(own[4 * i], own[4 * i + 1], own[4 * i + 2], own[4 * i + 3]);
            if (q != part) x = src[i * kBM3];
            sum[4 * i] += x.x; sum[4 * i + 1] += x.y; sum[4 * i + 2] += x.z; sum[4 * i + 3] += x.w;
          }
        }
        const int col = col0 + my_col + c;
        if (col < N) store_acc_chunk16<kF32Out>(c_out, row, ldc, col, sum);
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1 && !misaligned) {
    tc_fence_after();
    tmem_dealloc(tmem, tmem_cols);
  }
  // A CTA in which a wait ran out gets here while peers may still be sending, and storing into a
  // CTA that has left is a fault: it stays until every peer has left or stays as well, and these
  // have all issued their stores, and until the stores have landed. (Otherwise it has received
  // all parts and nobody stores into it any more. A barrier in every launch costs 0.5 us.)
  if (kSplit && !misaligned && *abort_flag != 0) {
    cluster_arrive();
    cluster_wait();   // for all threads of the cluster that have not left
    if (threadIdx.x == 0 && !mbar_try_wait(bar_parts, 0)) {
      const uint64_t t0 = globaltimer_ns();
      while (!mbar_try_wait(bar_parts, 0) && globaltimer_ns() - t0 < kWaitLimitNs) {}
    }
  }
}

template <int kBN, bool kF32Out, bool kSplit, bool kFold>
int launch_one3(const DeviceCtx& ctx, const GemmSplitPlan& p, const GemmSplitLayout& l, void* C, const void* A, const void* Bt, int groups, int M,
                int N, int K, int ldc, cudaStream_t stream) {
  CUtensorMap ta, tb;
  int rc = encode_tmap_bf16_2d(&ta, A, (uint64_t)groups * M, (uint64_t)K, (uint64_t)K * 2, kBM3, kBK3);
  if (rc != PTXB200_OK) return rc;
  rc = encode_tmap_bf16_2d(&tb, Bt, (uint64_t)groups * N, (uint64_t)K, (uint64_t)K * 2, kBN, kBK3);
  if (rc != PTXB200_OK) return rc;
  static PerDeviceOnce attr_once;
  rc = attr_once.run(ctx.device, []() -> int {
    PTXB200_CUDA_TRY(cudaFuncSetAttribute(gemm_split_kernel<kBN, kF32Out, kSplit, kFold>,
                                          cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax3));
    return PTXB200_OK;
  });
  if (rc != PTXB200_OK) return rc;
  const unsigned grid = (unsigned)(groups * (M / kBM3) * ((N + kBN - 1) / kBN) * p.split);
  PTXB200_CUDA_TRY(launch_after(stream, gemm_split_kernel<kBN, kF32Out, kSplit, kFold>, grid, kThreads3, (size_t)l.smem_bytes,
                                kSplit ? (unsigned)p.split : 1u, ta, tb, C, M, N, K, ldc, p.split, l.stages, l.chain_stages,
                                (uint32_t)l.tmem_cols, part_cols3(kBN, p.split), slot_bytes3(kBN, p.split), status_word(ctx, stream)));
  return PTXB200_OK;
}

template <int kBN, bool kF32Out, class... Args>
int launch_parts3(const DeviceCtx& ctx, const GemmSplitPlan& p, const GemmSplitLayout& l, Args... args) {
  if (p.split == 1) return launch_one3<kBN, kF32Out, false, false>(ctx, p, l, args...);
  return l.fold ? launch_one3<kBN, kF32Out, true, true>(ctx, p, l, args...)
                : launch_one3<kBN, kF32Out, true, false>(ctx, p, l, args...);
}

}  // namespace

void query_clusters(int sm_count, int (&clusters)[kMaxParts3 + 1]) {
  for (int& c : clusters) c = 0;
  clusters[1] = sm_count;
  auto* kernel = gemm_split_kernel<128, false, true, false>;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax3);
  for (int n = 2; n <= kMaxParts3 && e == cudaSuccess; ++n) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(sm_count / n * n));
    cfg.blockDim = dim3(kThreads3);
    cfg.dynamicSmemBytes = kSmemMax3;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim = {(unsigned)n, 1, 1};
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    e = cudaOccupancyMaxActiveClusters(&clusters[n], kernel, &cfg);
    if (e != cudaSuccess) clusters[n] = 0;
  }
  if (e != cudaSuccess) cudaGetLastError();   // clusters of two then
}

bool gemm_split_choose(const DeviceCtx& ctx, int groups, int M, int N, int K, unsigned flags, GemmSplitPlan* plan) {
  return gemm_split_rule(ctx.sm_count, ctx.clusters, groups, M, N, K / kBK3, (flags & PTXB200_GEMM_NO_SPLIT) == 0, plan);
}

int launch_gemm_split(const DeviceCtx& ctx, const GemmSplitPlan& p, void* C, const void* A, const void* Bt, int groups,
                      int M, int N, int K, int ldc, unsigned flags, cudaStream_t stream) {
  const bool f32 = (flags & PTXB200_GEMM_F32_OUT) != 0;
  const int kiters = K / kBK3;
  const int longest = (flags & PTXB200_GEMM_NO_SPLIT) ? 0 : gemm_line(ctx.sm_count, groups, M, N, kiters).share;
  const GemmSplitLayout l = gemm_split_layout(p, kiters, f32, longest);
  if (p.bn == 192)                    // always two parts, whose chains never fold
    return f32 ? launch_one3<192, true, true, false>(ctx, p, l, C, A, Bt, groups, M, N, K, ldc, stream)
               : launch_one3<192, false, true, false>(ctx, p, l, C, A, Bt, groups, M, N, K, ldc, stream);
  if (p.bn == 64)
    return f32 ? launch_parts3<64, true>(ctx, p, l, C, A, Bt, groups, M, N, K, ldc, stream)
               : launch_parts3<64, false>(ctx, p, l, C, A, Bt, groups, M, N, K, ldc, stream);
  return f32 ? launch_parts3<128, true>(ctx, p, l, C, A, Bt, groups, M, N, K, ldc, stream)
             : launch_parts3<128, false>(ctx, p, l, C, A, Bt, groups, M, N, K, ldc, stream);
}

}  // namespace ptxb200
