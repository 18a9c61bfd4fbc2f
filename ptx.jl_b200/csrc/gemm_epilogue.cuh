// Accumulator -> C stores shared by the GEMM kernels, as fp32 or rounded to bf16, in 128-bit
// stores.
//
// store_acc_16x64 takes 16 rows x 64 columns in the fragments that a 16-lane load of tensor
// memory delivers and exchanges words within quads of lanes, so that a quad writes 64
// consecutive bytes of a row and an instruction touches 8 rows. With a row per lane it touched
// 32, and the stores of a 256x256 tile kept its warps busy for 3.4 us, more than the products
// of K = 512 take: 4096x4096x256 18.2 us, now 15.3; 3072x3072x1024 with fp32 output 27.5 and 19.9.
#pragma once
#include "sm100_prims.cuh"

namespace ptxb200 {

// Rows row, row + 8 (this lane's two: row = the first of the 16 + lane / 4), columns col .. col + 63.
template <bool kF32Out>
__device__ __forceinline__ void store_acc_16x64(void* __restrict__ c_out, size_t row, int ldc, int col,
                                                const uint32_t (&o)[32]) {
  const int j = threadIdx.x & 3;
  if (kF32Out) {
    // lanes 0, 2 of a quad take columns 0-3, 4-7 of an even block of 8, lanes 1, 3 of the odd one behind it
    const bool odd = (j & 1) != 0;
    float* dst = reinterpret_cast<float*>(c_out) + row * (size_t)ldc + col + 8 * (j & 1) + 4 * (j >> 1);
#pragma unroll
    for (int p = 0; p < 4; ++p) {
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const uint32_t e0 = o[8 * p + 2 * r], e1 = o[8 * p + 2 * r + 1];           // even block
        const uint32_t d0 = o[8 * p + 4 + 2 * r], d1 = o[8 * p + 4 + 2 * r + 1];   // odd block
        const uint32_t x0 = __shfl_xor_sync(0xffffffffu, odd ? e0 : d0, 1);
        const uint32_t x1 = __shfl_xor_sync(0xffffffffu, odd ? e1 : d1, 1);
        st_global_v4(dst + (size_t)(8 * r) * ldc + 16 * p, odd ? x0 : e0, odd ? x1 : e1, odd ? d0 : x0, odd ? d1 : x1);
      }
    }
  } else {
    __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(c_out) + row * (size_t)ldc + col + 8 * j;
#pragma unroll
    for (int m = 0; m < 2; ++m) {
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        uint32_t w[4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
          w[i] = pack_bf16x2(__uint_as_float(o[4 * (4 * m + i) + 2 * r]), __uint_as_float(o[4 * (4 * m + i) + 2 * r + 1]));
        quad_transpose(w[0], w[1], w[2], w[3]);
        st_global_v4(dst + (size_t)(8 * r) * ldc + 32 * m, w[0], w[1], w[2], w[3]);
      }
    }
  }
}

// One row per lane, 16 consecutive columns.
template <bool kF32Out>
__device__ __forceinline__ void store_acc_chunk16(void* __restrict__ c_out, size_t row, int ldc, int col,
                                                  const float (&v)[16]) {
  if (kF32Out) {
    float* dst = reinterpret_cast<float*>(c_out) + row * (size_t)ldc + col;
#pragma unroll
    for (int i = 0; i < 4; ++i)
      st_global_v4(dst + 4 * i, __float_as_uint(v[4 * i]), __float_as_uint(v[4 * i + 1]), __float_as_uint(v[4 * i + 2]),
                   __float_as_uint(v[4 * i + 3]));
  } else {
    __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(c_out) + row * (size_t)ldc + col;
#pragma unroll
    for (int i = 0; i < 2; ++i)
      st_global_v4(dst + 8 * i, pack_bf16x2(v[8 * i], v[8 * i + 1]), pack_bf16x2(v[8 * i + 2], v[8 * i + 3]),
                   pack_bf16x2(v[8 * i + 4], v[8 * i + 5]), pack_bf16x2(v[8 * i + 6], v[8 * i + 7]));
  }
}

}  // namespace ptxb200
