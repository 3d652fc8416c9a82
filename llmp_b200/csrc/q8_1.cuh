// A Q8_1 block (36 bytes: FP16 d, FP16 sum of the inputs, 32 int8) by eight lanes of a warp.
#ifndef LLMP_B200_CSRC_Q8_1_CUH_
#define LLMP_B200_CSRC_Q8_1_CUH_

#include <cuda_fp16.h>

#include "common.cuh"

namespace llmp_b200 {

// Lane lane8 holds values 4 lane8 .. 4 lane8 + 3; whole warps call it; `live` lanes (whole groups of eight)
// store to the block at o.
__device__ __forceinline__ void QuantizeQ8_1Lane(const float (&v)[4], int lane8, bool live, std::uint8_t* o) {
  float amax = fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3])));
  float s[4] = {v[0], v[1], v[2], v[3]};
#pragma unroll
  for (int offset = 4; offset > 0; offset >>= 1) {
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, offset));
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      s[c] = s[c] + __shfl_xor_sync(0xffffffffu, s[c], offset);
    }
  }
  const float sum = (s[0] + s[2]) + (s[1] + s[3]);
  const float d = amax / 127.0f;
  std::uint32_t packed = 0;
  if (amax != 0.0f) {
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int q = static_cast<int>(roundf(v[c] / d));
      packed |= (static_cast<std::uint32_t>(q) & 0xffu) << (8 * c);
    }
  }
  if (!live) return;
  *reinterpret_cast<std::uint32_t*>(o + 4 + (lane8 * 4)) = packed;
  if (lane8 == 0) {
    const std::uint32_t ds = static_cast<std::uint32_t>(__half_as_ushort(__float2half_rn(d))) |
                             (static_cast<std::uint32_t>(__half_as_ushort(__float2half_rn(sum)))
                              << 16);
    *reinterpret_cast<std::uint32_t*>(o) = ds;
  }
}

}  // namespace llmp_b200

#endif  // LLMP_B200_CSRC_Q8_1_CUH_
