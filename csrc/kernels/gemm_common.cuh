// Pieces shared by the one-CTA and the CTA-pair grouped GEMM kernels: tile walk and epilogues.
#pragma once
#include "api.h"
#include "sm100_ptx.cuh"
#include "tile_walker.h"

namespace fastb {
namespace gemm {

constexpr int BN = 256, BK = 64, UMMA_K = 16;

static_assert(BK == kWalkBK, "the tile walker counts reduction steps of BK");

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&v);
}
// 1 / (1 + exp(-x)) and x times that. Built with --use_fast_math (FASTB_FAST_MATH): two operations of the special-function unit; a division, approximate
// too, takes more of them, for divisors above 2^126, whose reciprocal is zero anyway. Built without: the rounded division.
#ifdef FASTB_FAST_MATH
__device__ __forceinline__ float sigmoid(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(1.0f + __expf(-x)));
  return r;
}
__device__ __forceinline__ float silu(float x) { return x * sigmoid(x); }
#else
__device__ __forceinline__ float sigmoid(float x) { return 1.0f / (1.0f + __expf(-x)); }
__device__ __forceinline__ float silu(float x) { return x / (1.0f + __expf(-x)); }
#endif
__device__ __forceinline__ uint4 pack8(const uint32_t* r) {
  return make_uint4(pack_bf16(__uint_as_float(r[0]), __uint_as_float(r[1])), pack_bf16(__uint_as_float(r[2]), __uint_as_float(r[3])),
                    pack_bf16(__uint_as_float(r[4]), __uint_as_float(r[5])), pack_bf16(__uint_as_float(r[6]), __uint_as_float(r[7])));
}

// One thread = one output row: reads its 256 fp32 accumulators from TMEM (t_row = TMEM address of
// the row's first column) and writes bf16 to global. `zero` writes zeros without touching TMEM.
__device__ __forceinline__ void epilogue_store_row(__nv_bfloat16* crow, uint32_t t_row, bool zero) {
#pragma unroll 1
  for (int c = 0; c < BN / 32; ++c) {
    uint32_t r[32];
    if (!zero) { ptx::tmem_ld_32x32(t_row + c * 32, r); ptx::tmem_wait_ld(); }
    else {
#pragma unroll
      for (int i = 0; i < 32; ++i) r[i] = 0;
    }
    uint4* dst = reinterpret_cast<uint4*>(crow + c * 32);
#pragma unroll
    for (int q = 0; q < 4; ++q) dst[q] = pack8(r + 8 * q);
  }
}

// SwiGLU: the 256 columns of a tile are [128 gate | 128 up] of the same 128 features.
__device__ __forceinline__ void epilogue_swiglu_row(__nv_bfloat16* arow, __nv_bfloat16* gurow, uint32_t t_row) {
#pragma unroll 1
  for (int c = 0; c < BN / 64; ++c) {
    uint32_t g[32], u[32];
    ptx::tmem_ld_32x32(t_row + c * 32, g);
    ptx::tmem_ld_32x32(t_row + BN / 2 + c * 32, u);
    ptx::tmem_wait_ld();
    uint4* dst = reinterpret_cast<uint4*>(arow + c * 32);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      float o[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) o[i] = silu(__uint_as_float(g[8 * q + i])) * __uint_as_float(u[8 * q + i]);
      dst[q] = make_uint4(pack_bf16(o[0], o[1]), pack_bf16(o[2], o[3]), pack_bf16(o[4], o[5]), pack_bf16(o[6], o[7]));
    }
    if (gurow) {
      uint4* dg = reinterpret_cast<uint4*>(gurow + c * 32);
      uint4* du = reinterpret_cast<uint4*>(gurow + BN / 2 + c * 32);
#pragma unroll
      for (int q = 0; q < 4; ++q) { dg[q] = pack8(g + 8 * q); du[q] = pack8(u + 8 * q); }
    }
  }
}

}  // namespace gemm
}  // namespace fastb
