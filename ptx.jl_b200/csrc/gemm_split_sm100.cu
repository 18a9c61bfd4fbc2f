// gemm_bf16 for products with too few large tiles to fill the machine: one 128-row tile of
// 64 or 128 columns per CTA, with K split over the 1, 2 or 4 CTAs of a cluster.
//
// What bounds such a product is not the tensor pipe but one CTA's chain: launch, tensor
// maps, first loads, then about 0.16 us (64 columns) or 0.19 us (128) per 64 steps of K --
// shared memory takes in and feeds out 24 or 32 KiB per step -- and the epilogue. So the
// work is spread over as many CTAs as there are SMs: small tiles first, then K. The parts
// of a tile meet inside the cluster: every CTA sends each other one its share of the
// columns of the partial sums with asynchronous stores into that CTA's shared memory
// (counted on an mbarrier there), adds up its own share in the order of the parts, and
// writes it. Nothing goes through global memory, there is no second kernel, and no CTA
// waits for one that the hardware has not co-scheduled with it. The order of the sums is
// fixed, so results are reproducible (they differ in the last bits from the unsplit order).
// One-shot blocks: the first loads are issued before the block's threads even meet.
//
// With fp32 output a CTA sums its part of K in chains of at most 8 steps, up to 8 chains (64
// columns) or 4 (128), one accumulator in tensor memory each, and adds them up in the epilogue: the
// tensor core's fp32 accumulation loses about 3e-8 of the result per step of a chain, so
// one chain over 64 steps (1024x1152x8192 split in 2) is off by 4.0e-6, four of 16 steps by
// 8.5e-7 (the 35-step shares of the schedule before: 1.9e-6). bf16 output rounds 1.7e-3.
//
// Measured (device time, bf16 out unless noted; before: 128x256 tiles cut into shares of
// one k-iteration line, partial tiles parked in global memory, a second kernel to add
// them up): 128x4096x4096 20.4 -> 12.5 us; 1024x1152x8192 fp32 out 33.5 -> 21.0; 1024^3
// 14.6 -> 6.7; 512^3 7.9 -> 4.9; 128x128x8192 16.6 -> 9.9.
//
// Algorithmic work per launch: 2*G*M*N*K flop; compulsory bytes G*((M*K + N*K)*2 +
// M*N*sizeof(out)).
#include "cta_pair.cuh"
#include "gemm_epilogue.cuh"
#include "host_common.h"

namespace ptxb200 {
namespace {

constexpr int kBM3 = 128;
constexpr int kBK3 = 64;              // one 128-byte swizzle row of bf16
constexpr int kThreads3 = 192;        // warp 0 TMA producer, warp 1 MMA, warps 2-5 epilogue
constexpr int kMaxStages3 = 7;
constexpr int kSmemMax3 = 232448;
constexpr int kABytes3 = kBM3 * kBK3 * 2;
constexpr int kBandM3 = 8;            // row-tiles per rasterisation band
constexpr int kChainSteps3 = 8;       // steps of K per accumulator with fp32 output, more only where accumulators run out
// full[], empty[], acc_full, parts_in, TMEM slot, abort flag
constexpr int kCtrlBytes3 = ((2 * kMaxStages3 + 2) * 8 + 8 + 15) / 16 * 16;
static_assert(kCtrlBytes3 % 16 == 0, "the parts handed over behind it are 16-byte pieces");

enum : uint32_t { kSite3Empty = 24, kSite3Full = 25, kSite3AccFull = 26, kSite3Parts = 27 };

// steps of K per ring stage: two of 24 KiB (64 columns), or one of 32 KiB
__host__ __device__ constexpr int stage_k3(int bn) { return bn == 64 ? 2 : 1; }
__host__ __device__ constexpr int stage_bytes3(int bn) { return stage_k3(bn) * (kABytes3 + bn * kBK3 * 2); }
// what the other parts of the tile hand a CTA: [split - 1][bn / split / 4][128 rows] float4
__host__ __device__ constexpr int recv_bytes3(int bn, int split) { return (split - 1) * kBM3 * (bn / split) * 4; }

// 16 columns of this thread's row, summed over the chains (accumulators kBN columns apart)
template <int kBN>
__device__ __forceinline__ void load_sum16(uint32_t taddr, int chains, float (&x)[16]) {
  uint32_t v[16];
  tmem_ld16(taddr, v);
  tc_wait_ld_bind16(v);
#pragma unroll
  for (int i = 0; i < 16; ++i) x[i] = __uint_as_float(v[i]);
#pragma unroll 1
  for (int a = 1; a < chains; ++a) {
    tmem_ld16(taddr + a * kBN, v);
    tc_wait_ld_bind16(v);
#pragma unroll
    for (int i = 0; i < 16; ++i) x[i] += __uint_as_float(v[i]);
  }
}

template <int kBN, bool kF32Out>
__global__ void __launch_bounds__(kThreads3, 1)
gemm_split_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                  void* __restrict__ c_out, int M, int N, int K, int ldc, int split, int stages, int chain_stages,
                  uint32_t tmem_cols, uint32_t* status) {
  constexpr int kStageK = stage_k3(kBN), kStageBytes = stage_bytes3(kBN);
  constexpr int kAtomBytes = kABytes3 + kBN * kBK3 * 2;
  extern __shared__ __align__(1024) uint8_t smem[];
  const uint32_t base = smem_u32(smem);
  const int part = split > 1 ? (int)cluster_ctarank() : 0;   // which part of K this CTA of the cluster sums

  const uint32_t ctrl = base + stages * kStageBytes;
  uint8_t* ctrl_ptr = smem + stages * kStageBytes;
  const uint32_t bar_full = ctrl, bar_empty = ctrl + 8 * kMaxStages3, bar_acc = ctrl + 16 * kMaxStages3;
  const uint32_t bar_parts = bar_acc + 8;
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(ctrl_ptr + 16 * kMaxStages3 + 16);
  volatile uint32_t* abort_flag = tmem_slot + 1;
  const uint32_t recv = ctrl + kCtrlBytes3;
  const float4* recv_ptr = reinterpret_cast<const float4*>(ctrl_ptr + kCtrlBytes3);
  const WaitCtx wctx{status, abort_flag};

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const bool misaligned = (base & 1023u) != 0;   // the swizzled tiles need a 1024-byte aligned base
  if (misaligned && threadIdx.x == 0 && status != nullptr) atomicCAS(status, 0u, kStatusTimeoutTag | (17u << 8));

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
  const int k0 = (int)((long long)kiters * part / split), k1 = (int)((long long)kiters * (part + 1) / split);
  const int steps = (k1 - k0 + kStageK - 1) / kStageK;       // ring stages this CTA fills; the last may be a half

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
    mbar_init(bar_acc, 1);
    mbar_init(bar_parts, 1);
    mbar_fence_init();
    if (split > 1) mbar_arrive_expect_tx(bar_parts, recv_bytes3(kBN, split));
    if (!misaligned)
      for (int i = 0; i < stages && i < steps; ++i) load(i, i);
  }
  if (warp == 1 && !misaligned) {
    tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_slot)), tmem_cols);
    tmem_relinquish();
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (split > 1) cluster_arrive();          // "this CTA has started": waited for ahead of the first store to a peer
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
    }
    __syncwarp();
  } else if (!misaligned && warp == 1) {
    constexpr uint32_t idesc = make_idesc_bf16_f32(kBM3, kBN, false, false);
    constexpr uint32_t dhi = sdesc_hi(1024, kLayoutB128);
    int s = 0;
    uint32_t ph = 0, acc = tmem, first = 0;     // the chain's accumulator; 0: its first product overwrites it
    int left = chain_stages;                    // stages until the next chain begins
    auto mma = [&](int a, int slot, uint32_t accumulate) {   // one step of K: 4 instructions of 16
      const uint32_t da = sdesc_lo(base + slot * kStageBytes + a * kAtomBytes, 16);
      const uint32_t db = sdesc_lo(base + slot * kStageBytes + a * kAtomBytes + kABytes3, 16);
#pragma unroll
      for (int kk = 0; kk < kBK3 / 16; ++kk)   // 2 descriptor units = 32 bytes = 16 elements of K
        tc_mma_ss_warp(acc, da + 2 * kk, dhi, db + 2 * kk, dhi, idesc, kk == 0 ? accumulate : 1u);
    };
    // full stages first, without a branch around any instruction (one in this loop costs
    // about a hundred cycles a step), then a last half stage
    const int full_steps = (k1 - k0) / kStageK;
    for (int i = 0; i < full_steps; ++i) {
      mbar_wait_warp(bar_full + 8 * s, ph, wctx, kSite3Full);
      tc_fence_after();
      mma(0, s, first);
      if constexpr (kStageK == 2) mma(1, s, 1u);
      tc_commit_warp(bar_empty + 8 * s);
      if (++s == stages) { s = 0; ph ^= 1u; }
      const bool next = --left == 0;
      first = next ? 0u : 1u;
      acc += next ? (uint32_t)kBN : 0u;
      left = next ? chain_stages : left;
    }
    if (full_steps < steps) {
      mbar_wait_warp(bar_full + 8 * s, ph, wctx, kSite3Full);
      tc_fence_after();
      mma(0, s, first);
    }
    tc_commit_warp(bar_acc);
  }

  const int quad = warp & 3;
  const int row_in_tile = quad * 32 + lane;
  const bool epilogue = warp >= 2 && !misaligned;
  const uint32_t t_row = tmem_addr(tmem, quad * 32, 0);
  const size_t row = (size_t)g * M + (size_t)tm * kBM3 + row_in_tile;
  const int col0 = tn * kBN;
  const int chains = kF32Out ? (steps + chain_stages - 1) / chain_stages : 1;
  if (epilogue) {
    mbar_wait(bar_acc, 0, wctx, kSite3AccFull);
    tc_fence_after();
  }
  if (split == 1) {
    if (epilogue) {
#pragma unroll 1
      for (int h = 0; h < 2; ++h) {          // this warp's first and second 16 rows
        const size_t row16 = (size_t)g * M + (size_t)tm * kBM3 + quad * 32 + h * 16 + (lane >> 2);
#pragma unroll 1
        for (int c = 0; c < kBN; c += 64) {
          uint32_t v[32];
          tmem_ld_16x64(t_row + ((uint32_t)(h * 16) << 16) + c, v);
          tc_wait_ld_bind(v);
#pragma unroll 1
          for (int a = 1; a < chains; ++a) {
            uint32_t x[32];
            tmem_ld_16x64(t_row + ((uint32_t)(h * 16) << 16) + a * kBN + c, x);
            tc_wait_ld_bind(x);
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) + __uint_as_float(x[i]));
          }
          if (col0 + c < N) store_acc_16x64<kF32Out>(c_out, row16, ldc, col0 + c, v);   // N % 64 == 0
        }
      }
    }
  } else {
    // every part sums up and writes bn / split columns: it sends the others theirs
    const int width = kBN / split;
    cluster_wait();
    if (epilogue) {
#pragma unroll 1
      for (int i = 1; i < split; ++i) {
        const int q = part + i < split ? part + i : part + i - split;
        const uint32_t slot = part < q ? part : part - 1;
        const uint32_t dst = map_to_cta(recv + slot * (kBM3 * width * 4), q) + row_in_tile * 16;
        const uint32_t dst_bar = map_to_cta(bar_parts, q);
#pragma unroll 2
        for (int c = 0; c < width; c += 16) {
          float x[16];
          load_sum16<kBN>(t_row + q * width + c, chains, x);
#pragma unroll
          for (int j = 0; j < 4; ++j)
            st_async_v4(dst + (c / 4 + j) * (kBM3 * 16), dst_bar, x[4 * j], x[4 * j + 1], x[4 * j + 2], x[4 * j + 3]);
        }
      }
    }
    if (epilogue) {
      mbar_wait<true>(bar_parts, 0, wctx, kSite3Parts);   // other CTAs' stores are read behind it
#pragma unroll 1
      for (int c = 0; c < width; c += 16) {
        float own[16], sum[16];
        load_sum16<kBN>(t_row + part * width + c, chains, own);
#pragma unroll
        for (int i = 0; i < 16; ++i) sum[i] = 0.0f;
        // in the order of the parts, whoever adds them up
#pragma unroll 1
        for (int q = 0; q < split; ++q) {
          const float4* src = recv_ptr + (size_t)(q < part ? q : q - 1) * (kBM3 / 4 * width) + (c / 4) * kBM3 + row_in_tile;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            float4 x = make_float4(own[4 * i], own[4 * i + 1], own[4 * i + 2], own[4 * i + 3]);
            if (q != part) x = src[i * kBM3];
            sum[4 * i] += x.x; sum[4 * i + 1] += x.y; sum[4 * i + 2] += x.z; sum[4 * i + 3] += x.w;
          }
        }
        const int col = col0 + part * width + c;
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
  if (split > 1 && !misaligned && *abort_flag != 0) {
    cluster_arrive();
    cluster_wait();   // for all threads of the cluster that have not left
    if (threadIdx.x == 0 && !mbar_try_wait(bar_parts, 0)) {
      const uint64_t t0 = globaltimer_ns();
      while (!mbar_try_wait(bar_parts, 0) && globaltimer_ns() - t0 < kWaitLimitNs) {}
    }
  }
}

template <int kBN, bool kF32Out>
int launch_one3(const DeviceCtx& ctx, int split, void* C, const void* A, const void* Bt, int groups, int M, int N, int K,
                int ldc, bool one_chain, cudaStream_t stream) {
  CUtensorMap ta, tb;
  int rc = encode_tmap_bf16_2d(&ta, A, (uint64_t)groups * M, (uint64_t)K, (uint64_t)K * 2, kBM3, kBK3);
  if (rc != PTXB200_OK) return rc;
  rc = encode_tmap_bf16_2d(&tb, Bt, (uint64_t)groups * N, (uint64_t)K, (uint64_t)K * 2, kBN, kBK3);
  if (rc != PTXB200_OK) return rc;
  static PerDeviceOnce attr_once;
  rc = attr_once.run(ctx.device, []() -> int {
    PTXB200_CUDA_TRY(cudaFuncSetAttribute(gemm_split_kernel<kBN, kF32Out>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          kSmemMax3));
    return PTXB200_OK;
  });
  if (rc != PTXB200_OK) return rc;
  // a ring as deep as shared memory allows, but no deeper than the work
  const int recv = recv_bytes3(kBN, split);
  const int steps = ((K / kBK3 + split - 1) / split + stage_k3(kBN) - 1) / stage_k3(kBN);   // of the longest part
  int stages = (kSmemMax3 - kCtrlBytes3 - recv) / stage_bytes3(kBN);
  if (stages > kMaxStages3) stages = kMaxStages3;
  if (stages > steps) stages = steps;
  // chains of at most kChainSteps3 steps, as far as tensor memory holds accumulators
  int chains = one_chain || !kF32Out ? 1 : (steps * stage_k3(kBN) + kChainSteps3 - 1) / kChainSteps3;
  if (chains > 512 / kBN) chains = 512 / kBN;
  const int chain_stages = (steps + chains - 1) / chains;
  uint32_t tmem_cols = kBN;
  while (tmem_cols < (uint32_t)(chains * kBN)) tmem_cols *= 2;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(groups * (M / kBM3) * ((N + kBN - 1) / kBN) * split));
  cfg.blockDim = dim3(kThreads3);
  cfg.dynamicSmemBytes = (size_t)stages * stage_bytes3(kBN) + kCtrlBytes3 + recv;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim = {(unsigned)split, 1, 1};
  cfg.attrs = attr;
  cfg.numAttrs = split > 1 ? 1 : 0;
  PTXB200_CUDA_TRY(cudaLaunchKernelEx(&cfg, gemm_split_kernel<kBN, kF32Out>, ta, tb, C, M, N, K, ldc, split, stages,
                                      chain_stages, tmem_cols, status_word(ctx, stream)));
  return PTXB200_OK;
}

}  // namespace

// Which products run here, and how: those whose 128x128 tiles fit the SMs in one round (more
// tiles are better off in the persistent kernels: 2048x2048x512 9.1 us there, 9.1-11.2 here).
// Tiles of 64 columns if those fit too, since a step of K costs a CTA nearly the same for
// 64 columns as for 128 (1024^3: 6.7 against 7.7 us). K is split where SMs are left over and a
// part keeps at least 4 (split in 4) or 8 (in 2) steps: handing the parts over costs
// 1-2 us (384x640x1024: 5.8 in 4 parts, 6.7 whole; 512^3: 5.4 in 2 or 4 parts, 4.9 whole).
// Half of K on tiles of 128 columns against all of it on tiles of 64, which use equally
// many CTAs, pays from about 64 steps on (1024x1152: 16.1 against 16.5 us at 64 steps, 21.0
// against 25.3 at 128, 11.7 against 10.5 at 32).
bool gemm_split_choose(const DeviceCtx& ctx, int groups, int M, int N, int K, unsigned flags, GemmSplitPlan* plan) {
  const long long sms = ctx.sm_count, rows = (long long)groups * (M / kBM3);
  const long long tiles128 = rows * ((N + 127) / 128), tiles64 = rows * ((N + 63) / 64);
  if (tiles128 > sms) return false;
  const int kiters = K / kBK3;
  const bool may_split = !(flags & PTXB200_GEMM_NO_SPLIT);
  plan->split = 1;
  if (tiles64 > sms || (may_split && kiters >= 64 && tiles64 * 2 > sms && tiles128 * 2 <= sms)) {
    plan->bn = 128;
    if (may_split && kiters >= 16 && tiles128 * 2 <= sms) plan->split = 2;
    return true;
  }
  plan->bn = 64;
  if (may_split && kiters >= 16) plan->split = tiles64 * 4 <= sms ? 4 : tiles64 * 2 <= sms ? 2 : 1;
  return true;
}

int launch_gemm_split(const DeviceCtx& ctx, const GemmSplitPlan& p, void* C, const void* A, const void* Bt, int groups,
                      int M, int N, int K, int ldc, unsigned flags, cudaStream_t stream) {
  const bool f32 = (flags & PTXB200_GEMM_F32_OUT) != 0, one_chain = (flags & PTXB200_GEMM_NO_SPLIT) != 0;
  if (p.bn == 64)
    return f32 ? launch_one3<64, true>(ctx, p.split, C, A, Bt, groups, M, N, K, ldc, one_chain, stream)
               : launch_one3<64, false>(ctx, p.split, C, A, Bt, groups, M, N, K, ldc, one_chain, stream);
  return f32 ? launch_one3<128, true>(ctx, p.split, C, A, Bt, groups, M, N, K, ldc, one_chain, stream)
             : launch_one3<128, false>(ctx, p.split, C, A, Bt, groups, M, N, K, ldc, one_chain, stream);
}

}  // namespace ptxb200
