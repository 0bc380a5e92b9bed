// Epilogue steps shared by the grouped GEMMs that hold weight rows in TMEM lanes and tokens in TMEM columns: a thread
// owns one output column n of 32 tokens at a time (r[k] = token k).  Neighbouring lanes swap values, so that a lane ends
// up with neighbouring columns of one token and a warp stores whole 32-byte sectors of the tokens' rows.
#pragma once
#include <cstdint>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace rbv {
namespace tokepi {

__device__ __forceinline__ float silu(float x) { return x / (1.0f + __expf(-x)); }

// Lanes 2 j / 2 j + 1 hold gate j / up j of tokens k and k + 1: even lanes get silu(gate) * up of token k, odd lanes
// that of token k + 1.
__device__ __forceinline__ float swiglu_pair(const uint32_t (&r)[32], int k, bool odd) {
  const float mine = __uint_as_float(odd ? r[k + 1] : r[k]);
  const float got = __shfl_xor_sync(0xffffffffu, __uint_as_float(odd ? r[k] : r[k + 1]), 1);
  return odd ? silu(got) * mine : silu(mine) * got;
}

// SwiGLU of 32 tokens, bf16: `rows` is the address of column 0 of token 0, `col` this warp's first output column,
// `live` the number of tokens that exist.
__device__ __forceinline__ void store_swiglu(const uint32_t (&r)[32], __nv_bfloat16* rows, int ldc, int col, int live,
                                             int lane) {
  const bool odd = (lane & 1) != 0, hi = (lane & 2) != 0;
  #pragma unroll
  for (int k = 0; k < 32; k += 4) {
    const float o0 = swiglu_pair(r, k, odd), o1 = swiglu_pair(r, k + 2, odd);   // output column j = lane / 2
    // lanes with an even j keep token k + (lane & 1), the others token k + 2 + (lane & 1): two columns each
    const float got = __shfl_xor_sync(0xffffffffu, hi ? o0 : o1, 2);
    const __nv_bfloat162 v = hi ? __floats2bfloat162_rn(got, o1) : __floats2bfloat162_rn(o0, got);
    const int tok = k + (hi ? 2 : 0) + (odd ? 1 : 0);
    if (tok < live) *reinterpret_cast<__nv_bfloat162*>(rows + (size_t)tok * ldc + col + (lane >> 2) * 2) = v;
  }
}

// 32 tokens as bf16.  `row_of(tok)` gives the address of column 0 of a token (called by all lanes, with a token index
// that differs between even and odd lanes).
template <typename RowOf>
__device__ __forceinline__ void store_plain(const uint32_t (&r)[32], RowOf&& row_of, int col, int live, int lane) {
  const bool odd = (lane & 1) != 0;
  #pragma unroll
  for (int k = 0; k < 32; k += 2) {
    const float mine = __uint_as_float(odd ? r[k + 1] : r[k]);
    const float got = __shfl_xor_sync(0xffffffffu, __uint_as_float(odd ? r[k] : r[k + 1]), 1);
    const __nv_bfloat162 v = odd ? __floats2bfloat162_rn(got, mine) : __floats2bfloat162_rn(mine, got);
    const int tok = k + (odd ? 1 : 0);
    __nv_bfloat16* row = row_of(tok);
    if (tok < live) *reinterpret_cast<__nv_bfloat162*>(row + col + (lane & ~1)) = v;
  }
}

}  // namespace tokepi
}  // namespace rbv
