// Pieces shared by the tensor-core forward and backward kernels: 16-bit packing, bounded warp-wide barrier waits, and the
// host side of the TMA tensor maps.
#pragma once
#include <cuda.h>
#include <cudaTypedefs.h>

#include "hbsa_common.cuh"
#include "sm100_ptx.cuh"

namespace hbsa {

template <bool BF16> __device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  uint32_t r;
  if (BF16) asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  else asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}

// One lane polls the mbarrier, the rest of the warp sleeps at the shuffle instead of spinning.
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, long long budget) {
  int ok = 1;
  if ((threadIdx.x & 31) == 0) ok = ptx::mbar_wait_bounded(bar, parity, abort_flag, budget) ? 1 : 0;
  return __shfl_sync(0xffffffffu, ok, 0) != 0;
}
// Barrier entry and parity for the c-th use of a two-entry barrier array.
__device__ __forceinline__ uint32_t bar_of(uint32_t base, int c) { return base + 8u * (uint32_t)(c & 1); }
__device__ __forceinline__ uint32_t par_of(int c) { return (uint32_t)(c >> 1) & 1u; }

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// cuTensorMapEncodeTiled of the loaded driver, or NULL.
EncodeTiledFn sm100_encode_fn();
// 3-D map over a [tokens, heads, headdim] 16-bit tensor: dims (headdim, heads, tokens), box (64, box_heads, box_tokens).
bool sm100_encode_map(EncodeTiledFn fn, CUtensorMap* map, bool bf16, const void* base, int headdim, int heads, int tokens,
                      long long s_tok, long long s_head, int box_heads, int box_tokens);
int sm100_sm_count();
long long sm100_wait_budget();
int sm100_debug_stall();

}  // namespace hbsa
