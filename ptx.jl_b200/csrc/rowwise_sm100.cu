// Row-wise fp32 kernels either side of attention in a transformer block: softmax,
// RMS norm, layer norm (one output row from one input row) and SwiGLU (elementwise).
//
// The reference ships these as one-CTA-per-row kernels with the row held in
// registers between the reduction passes (test/gpu/softmax.jl:30-140,
// test/gpu/rms_norm.jl:30-106, test/gpu/layer_norm.jl:24-122,
// test/gpu/swiglu.jl:31-69): N must be a multiple of block*4 and at most
// block*64. All four are bound by HBM: 8 bytes per element (one fp32 read, one fp32
// write; the weight vectors stay in cache), 12 for SwiGLU.
//
// What is kept: one read of X, the row on chip across the passes, 128-bit accesses. What is
// different:
//   * one block per row (one per four rows with a warp each up to 2048 columns) and no loop
//     over rows in the kernel: a block that ends makes room for one whose loads start at
//     once, so reads and writes of different rows stay mixed. A persistent grid of the same
//     blocks falls into step (all read, then all write): rows of 8192 columns, 0.5 GB in,
//     0.5 GB out, softmax 171 us persistent, 156 us this way (6880 GB/s); rows of 1024
//     columns 91 against 80 us; and a ring in shared memory kept full by bulk copies 170 to 203;
//   * the threads per row follow its length, eight float4s each or four (any N that is a
//     multiple of 4: the last ones are guarded), in steps of a warp: rows of 9000 columns took
//     300 us on a power-of-two block that they half filled, and take 157;
//   * above 16384 columns a thread holds eight float4s in registers and up to eight in
//     shared memory, so that two blocks still fit an SM's register file and overlap
//     (softmax, 30000 columns: 197 us with the whole row in registers, 169 now);
//   * few rows (at most two per SM, up to 4096 columns) are spread over four times the
//     threads, and the weights are fetched ahead of the reduction: latency counts there (16
//     rows of 2048 columns, layer norm: 4.2 us, now 2.1); long ones over 1024 threads;
//   * X and Y are accessed with the streaming cache hints (read once, written once);
//   * a launch's blocks are set up while the kernel in front ends (launch_after): 300 rows of 2048
//     columns, back to back, 4.1 us a launch without, 2.4-2.75 with; 4096 x 30000, softmax, 158 and 156;
//   * softmax merges (max, sum of exponentials) pairs by the online-softmax rule and
//     rescales once; layer norm takes the mean, then the centred sums of the values on chip and
//     of their squares, which keeps its accuracy for rows with a large mean, where the
//     reference's E[x^2] - mean^2 cancels. With several warps per row a reduction costs one
//     block barrier.
#include "host_common.h"
#include "sm100_prims.cuh"

namespace ptxb200 {
namespace {

constexpr float kLog2e = 1.4426950408889634f;

enum RowOp : int { kOpSoftmax = 0, kOpRmsNorm = 1, kOpLayerNorm = 2 };

struct RowParams {
  float* y;
  const float* x;
  const float* w;      // rms_norm, layer_norm
  const float* bias;   // layer_norm
  int rows;
  int n4;              // N / 4
  float inv_n;
  float eps;
};

// Reductions over the threads that share a row: a sum, two sums, or a (max, sum of exponentials)
// pair merged with the online-softmax rule. With more than one warp per row the warps'
// partials meet in shared memory behind ONE block barrier: the buffer alternates between
// two from reduction to reduction, so a warp writing the next partials cannot overrun a
// reader of these (it would first have to pass a barrier which the reader also has to reach).
struct Pair { float m, s; };          // running max and sum of 2^((x - m) log2 e)

__device__ __forceinline__ Pair merge(Pair a, Pair b) {
  const float m = fmaxf(a.m, b.m);
  // a side that holds only padding has m = -inf and s = 0; (-inf) - (-inf) must not reach ex2
  const float fa = a.m == m ? 1.0f : ex2_approx((a.m - m) * kLog2e);
  const float fb = b.m == m ? 1.0f : ex2_approx((b.m - m) * kLog2e);
  return {m, a.s * fa + b.s * fb};
}
__device__ __forceinline__ float merge(float a, float b) { return a + b; }
struct Sums { float a, b; };
__device__ __forceinline__ Sums merge(Sums x, Sums y) { return {x.a + y.a, x.b + y.b}; }

__device__ __forceinline__ float shfl_xor(float v, int o) { return __shfl_xor_sync(0xffffffffu, v, o); }
__device__ __forceinline__ Pair shfl_xor(Pair v, int o) { return {shfl_xor(v.m, o), shfl_xor(v.s, o)}; }
__device__ __forceinline__ Sums shfl_xor(Sums v, int o) { return {shfl_xor(v.a, o), shfl_xor(v.b, o)}; }
__device__ __forceinline__ float identity(float) { return 0.0f; }
__device__ __forceinline__ Sums identity(Sums) { return {0.0f, 0.0f}; }
__device__ __forceinline__ Pair identity(Pair) { return {-INFINITY, 0.0f}; }

template <typename T>
__device__ __forceinline__ T warp_reduce(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = merge(v, shfl_xor(v, o));
  return v;
}

// Global loads stay behind grid_wait: they go through pointers that the compiler only knows behind
// it (behind). The weights are loaded plainly and not through the read-only path (ld.global.nc), which
// wants memory that nothing writes while this kernel runs: it starts ahead of the end of the kernel in
// front, which may be writing them. The compiler moves no plain load past a store, so that the
// weights of a thread's next groups are fetched ahead of the stores in the source (kAhead; 423 x 23104, layer
// norm: 19.7 us through the read-only path, 20.1 this way, 22.7 with each group's loads behind the store of the one
// before; 4096 x 30000 194, 194 and 204; RMS norm 161, 162 and 170).
// These kernels do not let their successor in early (grid_trigger): 4000 x 1024, layer norm, 7.2 us
// with it at the start of a block, 5.6 without.
__device__ __forceinline__ float4 load_once(const float4* p) {   // streaming: read once
  float4 v;
  asm("ld.global.cs.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ float4 load_shared_by_rows(const float4* p) {
  float4 v;
  asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  return v;
}
template <class T>
__device__ __forceinline__ const T* behind(const T* p) {
  asm volatile("" : "+l"(p)::"memory");
  return p;
}
__device__ __forceinline__ void cp_async16(uint32_t dst_smem, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst_smem), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// One row per block (kWarpRows = false: all threads of the block share it) or per warp
// (kWarpRows = true, four rows per block). A thread holds the row's float4s t, t + T, ...
// (T threads per row): the first kVec of them in registers, kPark more in shared memory
// slots that no other thread touches. Blocks have up to kMaxT threads, kMinBlocks of them fit an SM.
template <int kOp, bool kWarpRows, int kVec, int kPark, int kMaxT, int kMinBlocks>
__global__ void __launch_bounds__(kMaxT, kMinBlocks)
rowwise_kernel(const RowParams p) {
  __shared__ float2 red[2][32];
  extern __shared__ __align__(16) float4 parked[];   // [kPark][T]
  const int tpr = kWarpRows ? 32 : blockDim.x;       // threads per row
  const int t = kWarpRows ? threadIdx.x & 31 : threadIdx.x;
  const int row = kWarpRows ? blockIdx.x * 4 + (threadIdx.x >> 5) : blockIdx.x;
  grid_wait();
  if (kWarpRows && row >= p.rows) return;            // the last block's rows may be fewer; no block barrier follows
  const float4* x4 = behind(reinterpret_cast<const float4*>(p.x)) + (size_t)row * p.n4;
  float4* y4 = reinterpret_cast<float4*>(p.y) + (size_t)row * p.n4;
  const float4* w4 = behind(reinterpret_cast<const float4*>(p.w));
  const float4* b4 = behind(reinterpret_cast<const float4*>(p.bias));
  const float fill = kOp == kOpSoftmax ? -INFINITY : 0.0f;

  int parity = 0;
  auto reduce = [&](auto v) {
    v = warp_reduce(v);
    if constexpr (!kWarpRows) {
      decltype(v)* buf = reinterpret_cast<decltype(v)*>(red[parity]);
      parity ^= 1;
      if ((t & 31) == 0) buf[t >> 5] = v;
      __syncthreads();
      v = warp_reduce((t & 31) < (tpr >> 5) ? buf[t & 31] : identity(v));
    }
    return v;
  };

#pragma unroll
  for (int i = 0; i < kPark; ++i) {
    const int c = t + (kVec + i) * tpr;
    if (c < p.n4) cp_async16(smem_u32(parked + i * tpr + t), x4 + c);
    else parked[i * tpr + t] = make_float4(fill, fill, fill, fill);
  }
  float4 v[kVec];
#pragma unroll
  for (int i = 0; i < kVec; ++i) {
    const int c = t + i * tpr;
    v[i] = c < p.n4 ? load_once(x4 + c) : make_float4(fill, fill, fill, fill);
  }
  // The weights of the thread's first kAhead groups are fetched ahead of the last reduction (short shares:
  // of all, so that their latency does not follow it), the others' as these are written: as many as registers
  // allow (layer norm holds two vectors: with four ahead 2000 x 8192 takes 30 us, 23 with two).
  // A warp's rows: six, behind the reduction (layer norm, 65536 x 1024 78.5 us, 82 with all eight).
  constexpr bool kNorm = kOp != kOpSoftmax;
  constexpr int kAhead = kVec <= 2 ? kVec : kWarpRows ? (kVec < 6 ? kVec : 6) : kOp == kOpLayerNorm ? (kVec == 4 ? 1 : 2)
                         : kPark > 0 || kMaxT == 1024 ? 4 : 2;
  float4 w[kNorm ? kAhead : 1], b[kOp == kOpLayerNorm ? kAhead : 1];
  auto fetch_into = [&](int i, float4& wi, float4& bi) {
    const int c = t + i * tpr;
    if (c < p.n4) {
      wi = load_shared_by_rows(w4 + c);
      if constexpr (kOp == kOpLayerNorm) bi = load_shared_by_rows(b4 + c);
    }
  };
  auto fetch = [&](int i) { fetch_into(i, w[i % kAhead], b[kOp == kOpLayerNorm ? i % kAhead : 0]); };
  auto fetch_first = [&]() {
#pragma unroll
    for (int i = 0; i < kAhead; ++i) fetch(i);
  };
  if constexpr (kNorm && kVec <= 2) fetch_first();
  if (kPark > 0) cp_async_wait_all();

  // f(element group, its index in the row) over everything this thread holds
  auto each = [&](auto f) {
#pragma unroll
    for (int i = 0; i < kVec; ++i) f(v[i], t + i * tpr);
#pragma unroll 1
    for (int i = 0; i < kPark; ++i) {
      float4 x = parked[i * tpr + t];
      f(x, t + (kVec + i) * tpr);
      parked[i * tpr + t] = x;
    }
  };

  float mul;   // what the row's (centred, exponentiated) values are scaled by,
  [[maybe_unused]] float add;   // and layer norm: what is added then
  if constexpr (kOp == kOpSoftmax) {
    float m = -INFINITY;
    each([&](float4& x, int) { m = fmaxf(fmaxf(m, fmaxf(x.x, x.y)), fmaxf(x.z, x.w)); });
    // exponentials against this thread's own maximum, rescaled once the row's is known
    const float neg = m == -INFINITY ? 0.0f : -m * kLog2e;
    float s = 0.0f;
    each([&](float4& x, int) {
      x.x = ex2_approx(fmaf(x.x, kLog2e, neg));
      x.y = ex2_approx(fmaf(x.y, kLog2e, neg));
      x.z = ex2_approx(fmaf(x.z, kLog2e, neg));
      x.w = ex2_approx(fmaf(x.w, kLog2e, neg));
      s += (x.x + x.y) + (x.z + x.w);   // padding lanes hold 2^-inf = 0
    });
    const Pair tot = reduce(Pair{m, s});
    mul = (m == tot.m ? 1.0f : ex2_approx((m - tot.m) * kLog2e)) / tot.s;
  } else if constexpr (kOp == kOpRmsNorm) {
    float s = 0.0f;
    each([&](float4& x, int) { s += (x.x * x.x + x.y * x.y) + (x.z * x.z + x.w * x.w); });
    if constexpr (kVec > 2 && !kWarpRows) fetch_first();
    mul = rsqrtf(reduce(s) * p.inv_n + p.eps);
    if constexpr (kVec > 2 && kWarpRows) fetch_first();
  } else {
    // The mean is a sum in fp32 and off by its rounding, up to a few 1e-7 of itself. The mean of
    // the centred values is that error: it is taken off the values and, squared, off their mean
    // square. Rows around 1000 with unit spread: error 5.5e-5 without, 6e-8 with it; rows of one
    // value give zeros. (Each thread's sum is scaled ahead of the reduction, which then cannot
    // overflow where the mean does not.)
    float s = 0.0f;
    each([&](float4& x, int) { s += (x.x + x.y) + (x.z + x.w); });   // padding lanes hold zeros
    const float mean = reduce(s * p.inv_n);
    Sums d = {0.0f, 0.0f};
    each([&](float4& x, int c) {
      if (c < p.n4) {
        x.x -= mean; x.y -= mean; x.z -= mean; x.w -= mean;
        d.a += (x.x + x.y) + (x.z + x.w);
        d.b += (x.x * x.x + x.y * x.y) + (x.z * x.z + x.w * x.w);
      }
    });
    if constexpr (kVec > 2 && !kWarpRows) fetch_first();
    d = reduce(d);
    if constexpr (kVec > 2 && kWarpRows) fetch_first();
    const float off = d.a * p.inv_n;
    float var = d.b * p.inv_n;
    if (var < INFINITY) var = fmaxf(fmaf(-off, off, var), 0.0f);   // two rounded values: may cross zero (NaN: left alone)
    mul = rsqrtf(var + p.eps);
    add = -off * mul;
  }

  auto write = [&](const float4& x, int c, const float4& wi, const float4& bi) {
    float4 o;
    if constexpr (kOp == kOpLayerNorm)
      o = make_float4(fmaf(x.x, mul, add), fmaf(x.y, mul, add), fmaf(x.z, mul, add), fmaf(x.w, mul, add));
    else
      o = make_float4(x.x * mul, x.y * mul, x.z * mul, x.w * mul);
    if constexpr (kOp == kOpRmsNorm)
      o = make_float4(o.x * wi.x, o.y * wi.y, o.z * wi.z, o.w * wi.w);
    else if constexpr (kOp == kOpLayerNorm)
      o = make_float4(fmaf(o.x, wi.x, bi.x), fmaf(o.y, wi.y, bi.y), fmaf(o.z, wi.z, bi.z), fmaf(o.w, wi.w, bi.w));
    __stcs(y4 + c, o);
  };
  if constexpr (kOp == kOpSoftmax) {
#pragma unroll
    for (int i = 0; i < kVec; ++i) {
      const int c = t + i * tpr;
      if (c < p.n4) write(v[i], c, v[i], v[i]);
    }
    // (Two at a time: 4096 x 30000 155.5 us with four, 152.5 with two, 600 x 30000 29.5 and 27.5, 8000 x 24000
    // 236.6 and 229.3.)
#pragma unroll 2
    for (int i = 0; i < kPark; ++i) {
      const int c = t + (kVec + i) * tpr;
      if (c < p.n4) write(parked[i * tpr + t], c, v[0], v[0]);
    }
  } else {
    // Layer norm fetches a parked half four groups at a time, behind the stores of the first, whose
    // registers that takes; RMS norm goes on one by one (423 x 23104 17.3 us, 18.0 four at a time).
    constexpr int kRolling = kOp == kOpLayerNorm ? kVec : kVec + kPark;
#pragma unroll
    for (int i = 0; i < kRolling; ++i) {
      const int c = t + i * tpr;
      if (c < p.n4)
        write(i < kVec ? v[i < kVec ? i : 0] : parked[(i - kVec) * tpr + t], c, w[i % kAhead],
              b[kOp == kOpLayerNorm ? i % kAhead : 0]);
      if (i + kAhead < kRolling) fetch(i + kAhead);
    }
#pragma unroll 1
    for (int g = kRolling - kVec; g < kPark; g += 4) {
      float4 wg[4], bg[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) fetch_into(kVec + g + i, wg[i], bg[i]);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int c = t + (kVec + g + i) * tpr;
        if (c < p.n4) write(parked[(g + i) * tpr + t], c, wg[i], bg[i]);
      }
    }
  }
}

__device__ __forceinline__ float silu_mul(float g, float u) {
  // g * sigmoid(g) * u with exp(-g) = 2^(-g log2 e) (test/gpu/swiglu.jl:33-40)
  return g * rcp_approx(1.0f + ex2_approx(-g * kLog2e)) * u;
}

constexpr int kSwigluThreads = 256;

// kUnroll: independent 128-bit load pairs in flight per thread
template <int kUnroll>
__global__ void __launch_bounds__(kSwigluThreads)
swiglu_kernel(float* out, const float* gate, const float* up, size_t n4) {
  grid_wait();
  const float4* g4 = behind(reinterpret_cast<const float4*>(gate));
  const float4* u4 = behind(reinterpret_cast<const float4*>(up));
  float4* o4 = reinterpret_cast<float4*>(out);
  const size_t base = (size_t)blockIdx.x * (kSwigluThreads * kUnroll) + threadIdx.x;
  float4 g[kUnroll], u[kUnroll];
#pragma unroll
  for (int i = 0; i < kUnroll; ++i) {
    const size_t c = base + i * kSwigluThreads;
    if (c < n4) {
      g[i] = load_once(g4 + c);
      u[i] = load_once(u4 + c);
    }
  }
#pragma unroll
  for (int i = 0; i < kUnroll; ++i) {
    const size_t c = base + i * kSwigluThreads;
    if (c < n4)
      __stcs(o4 + c, make_float4(silu_mul(g[i].x, u[i].x), silu_mul(g[i].y, u[i].y), silu_mul(g[i].z, u[i].z),
                                 silu_mul(g[i].w, u[i].w)));
  }
}

template <int kOp, int kVec>
int launch_warp_rows(const RowParams& p, cudaStream_t stream) {
  PTXB200_CUDA_TRY(launch_after(stream, rowwise_kernel<kOp, true, kVec, 0, 128, 1>, (unsigned)((p.rows - 1) / 4 + 1), 128u, 0, 1u, p));
  return PTXB200_OK;
}

// A block per row, of as many threads as the row needs, in steps of a warp.
template <int kOp, int kVec, int kMaxT, int kMinBlocks, int kPark = 0>
int launch_block_rows(const RowParams& p, cudaStream_t stream) {
  constexpr int per = kVec + kPark;
  const int threads = kMaxT == 1024 ? 1024 : ((p.n4 + per - 1) / per + 31) / 32 * 32;
  PTXB200_CUDA_TRY(launch_after(stream, rowwise_kernel<kOp, false, kVec, kPark, kMaxT, kMinBlocks>, (unsigned)p.rows, (unsigned)threads,
                                (size_t)kPark * threads * 16, 1u, p));
  return PTXB200_OK;
}

// The lines lie where measured device times cross (inputs beyond L2); the norms, which fetch
// weights behind their reduction, want more threads per row than softmax.
template <int kOp>
int dispatch(const DeviceCtx& ctx, const RowParams& p, cudaStream_t stream) {
  const int n4 = p.n4;
  constexpr bool kNorm = kOp != kOpSoftmax;
  // At most two rows per SM: nothing overlaps, so a row's own latency is the launch's. 200 rows
  // of 2048 columns: 2.3 us against 2.6 with a warp per row (layer norm 2.4 against 4.4); above
  // 4096 columns the shorter chain per thread no longer pays (200 rows of 8192: 5.2 against 4.4).
  // Norms of 512 to 1024 columns up to eight rows per SM: layer norm, 1000 x 512 2.68 against
  // 3.11 with a warp per row, RMS norm, 600 x 1024 2.39 against 2.86.
  const bool few = p.rows <= 2 * ctx.sm_count;
  if (n4 <= 1024 && (few ? n4 >= (kNorm ? 128 : 129) : kNorm && n4 >= 128 && n4 <= 256 && p.rows <= 8 * ctx.sm_count))
    return launch_block_rows<kOp, 2, 512, 2>(p, stream);
  // At most one long row per SM: all of an SM's threads on it (148 x 20000, RMS norm: 5.9 us
  // against 7.0 with half in shared memory, layer norm 7.2 and 8.6, softmax 6.3 and 7.3).
  if (p.rows <= ctx.sm_count) {
    if (n4 > 4096) return launch_block_rows<kOp, 8, 1024, 1>(p, stream);
    if constexpr (kOp == kOpRmsNorm)
      if (n4 > 2048) return launch_block_rows<kOp, 4, 1024, 1>(p, stream);   // 148 x 12000: 4.4 against 4.9
  }
  // A warp per row; not for norms above 1024 columns (layer norm, 4000 x 2048: 14.5 us against
  // 12.0 on a block per row).
  if (n4 <= (kNorm ? 256 : 512)) {
    const int per = (n4 + 31) / 32;
    if (per <= 1) return launch_warp_rows<kOp, 1>(p, stream);
    if (per <= 2) return launch_warp_rows<kOp, 2>(p, stream);
    if (per <= 4) return launch_warp_rows<kOp, 4>(p, stream);
    if (kNorm || per <= 8) return launch_warp_rows<kOp, 8>(p, stream);
    if constexpr (!kNorm) return launch_warp_rows<kOp, 16>(p, stream);
  }
  // Four float4s per thread keep more rows in flight: RMS norm, 2000 x 4096 12.2 us with eight and
  // 11.5, 600 x 8192 9.1 and 8.5; layer norm, 4000 x 3000 17.3 and 16.8, but 2000 x 8192 23.0 and 24.2.
  if constexpr (kNorm)
    if (n4 <= (kOp == kOpRmsNorm || few ? 2048 : 1024)) return launch_block_rows<kOp, 4, 512, 3>(p, stream);
  if (n4 <= 8 * 512) return launch_block_rows<kOp, 8, 512, 2>(p, stream);
  static PerDeviceOnce attr_once;
  const int rc = attr_once.run(ctx.device, []() -> int {
    PTXB200_CUDA_TRY(cudaFuncSetAttribute(rowwise_kernel<kOp, false, 8, 8, 512, 2>,
                                          cudaFuncAttributeMaxDynamicSharedMemorySize, 512 * 8 * 16));
    return PTXB200_OK;
  });
  if (rc != PTXB200_OK) return rc;
  return launch_block_rows<kOp, 8, 512, 2, 8>(p, stream);
}

}  // namespace

int launch_rowwise(const DeviceCtx& ctx, int op, float* y, const float* x, const float* w,
                   const float* bias, int rows, int n, float eps, cudaStream_t stream) {
  RowParams p;
  p.y = y;
  p.x = x;
  p.w = w;
  p.bias = bias;
  p.rows = rows;
  p.n4 = n / 4;
  p.inv_n = 1.0f / (float)n;
  p.eps = eps;
  switch (op) {
    case kOpSoftmax: return dispatch<kOpSoftmax>(ctx, p, stream);
    case kOpRmsNorm: return dispatch<kOpRmsNorm>(ctx, p, stream);
    case kOpLayerNorm: return dispatch<kOpLayerNorm>(ctx, p, stream);
    default: return PTXB200_E_INVALID;
  }
}

int launch_swiglu(const DeviceCtx& ctx, float* out, const float* gate, const float* up, size_t n,
                  cudaStream_t stream) {
  const size_t n4 = n / 4;
  // one load pair per thread while that fits the machine in one round (2 us calls), else
  // four; blocks that each run once, for the same reason as above (65536 x 4096: 459 us
  // against 498 for a persistent grid)
  const bool small = n4 <= (size_t)ctx.sm_count * 8 * kSwigluThreads;
  const size_t per_block = (size_t)kSwigluThreads * (small ? 1 : 4);
  const size_t blocks = (n4 + per_block - 1) / per_block;
  if (blocks > 0x7fffffffu) return PTXB200_E_SHAPE;
  PTXB200_CUDA_TRY(launch_after(stream, small ? swiglu_kernel<1> : swiglu_kernel<4>, (unsigned)blocks, kSwigluThreads, 0, 1u, out, gate,
                                up, n4));
  return PTXB200_OK;
}

}  // namespace ptxb200
