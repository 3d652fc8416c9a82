// The unit of the dense token-column kernel (vecq_rowmma.cuh): 16 weight rows x one Q4_K super-block x
// up to eight tokens, one matrix, on mma.sync m16n8k32 (u8 x s8 -> s32).
//
//   * Eight tokens: the MMA's columns are the tokens, two MMAs a chunk of two sub-blocks, and a lane
//     folds 32 sums.  Up to four: the columns are tokens x the chunk's two sub-blocks, both MMAs into
//     one fragment (each lane's B is zero where its column is the other sub-block's), 16 sums a lane,
//     two thirds of the instructions.  The two add in the same order: the same bits.
//   * The fold is the multiply-add pipes' work: the MMA accumulates onto the bits of 1.5 * 2^23, so its
//     result is a float and one exact subtraction gives the sum; the 6-bit scale multiplies the token's
//     (17 bits, exact) and one multiply-add has the only rounding, d8 * sc * dot.  (A shift, a
//     conversion and an integer multiply are two cycles a warp instruction each, these one.)  Even and odd sub-blocks
//     are summed apart; the odd ones' codes stay in place as 16 x code and 1/16 goes to the token's
//     scale: both exact.
#ifndef LLMP_B200_CSRC_VECQ_COLUMNS_CUH_
#define LLMP_B200_CSRC_VECQ_COLUMNS_CUH_

#include "vecq_stream.cuh"

namespace llmp_b200 {
namespace vecq {

// Byte `i` of w as a float: 2^23 + it, less 2^23.
template <int i>
__device__ __forceinline__ float ByteFloat(std::uint32_t w) {
  return __uint_as_float(__byte_perm(w, 0x4b000000u, 0x7440u | i)) - 8388608.0f;
}

template <int i>
struct Index {
  static constexpr int value = i;
};

// The staged activations of up to kTokens tokens over `columns` super-block columns.
//   codes, per token: chunk by chunk (two sub-blocks), for t = 0..3 bytes 8t..8t+7 of the even
//   sub-block, then of the odd;
//   scales: eight tokens, per pair of tokens and sub-block (d8, d8, d8 * sum q, d8 * sum q);
//   four tokens, per token and chunk (d8, d8 / 16, d8 * sum q, d8 * sum q), even then odd.
template <int kTokens>
struct ColumnActs {
  int columns;
  __host__ __device__ constexpr explicit ColumnActs(int c) : columns(c) {}
  __host__ __device__ constexpr int Pitch() const { return (columns * 256) + 64; }
  __host__ __device__ constexpr int ScalePitch() const {
    return kTokens == 8 ? (columns * 128) + 32 : (columns * 64) + 16;
  }
  __host__ __device__ constexpr int Scales() const { return kTokens * Pitch(); }
  __host__ __device__ constexpr int Bytes() const { return (Scales() + (4 * ScalePitch()) + 127) / 128 * 128; }
};

template <int kTokens>
__device__ __forceinline__ void StageColumnBlock(unsigned char* acts, ColumnActs<kTokens> layout, int p, int b,
                                                const std::uint8_t* block) {
  const auto* src = reinterpret_cast<const std::uint32_t*>(block);
  std::uint32_t v[8];
  int isum = 0;
  const float d = HalfBitsToFloat(src[0] & 0xffffu);
#pragma unroll
  for (int w = 0; w < 8; ++w) {
    v[w] = src[1 + w];
    isum = Dp4a(0x01010101, static_cast<int>(v[w]), isum);
  }
  auto* codes = reinterpret_cast<uint2*>(acts + (p * layout.Pitch()) + ((b >> 1) * 64) + ((b & 1) * 8));
#pragma unroll
  for (int t = 0; t < 4; ++t) codes[2 * t] = make_uint2(v[2 * t], v[(2 * t) + 1]);
  float* scales = kTokens == 8
                      ? reinterpret_cast<float*>(acts + layout.Scales() + ((p >> 1) * layout.ScalePitch())) + (4 * b) + (p & 1)
                      : reinterpret_cast<float*>(acts + layout.Scales() + (p * layout.ScalePitch())) + (4 * (b >> 1)) + (b & 1);
  scales[0] = (b & 1) != 0 ? d * 0.0625f : d;
  scales[2] = d * static_cast<float>(isum);
}

// D = A * B onto the bits of 1.5 * 2^23 (|dot| < 2^22): a float 12582912 above the sum.
constexpr int kFloatBits = 0x4b400000;
__device__ __forceinline__ void MmaOnto(int (&d)[4], std::uint32_t a0, std::uint32_t a1, std::uint32_t a2,
                                        std::uint32_t a3, std::uint32_t b0, std::uint32_t b1, const int (&c)[4]) {
  asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
      "{%10, %11, %12, %13};"
      : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(c[0]), "r"(c[1]), "r"(c[2]), "r"(c[3]));
}
__device__ __forceinline__ float SumOf(int bits) { return __int_as_float(bits) - 12582912.0f; }

// The unit: rows g and g + 8 (blocks lo and hi) x column c of the staged ones.  Eight tokens: sums of
// tokens 2t and 2t + 1 a row; four: of token t.
template <int kTokens>
__device__ __forceinline__ void ColumnUnit(const unsigned char* lo, const unsigned char* hi,
                                          const unsigned char* codes, const unsigned char* scales, int lane, int c,
                                          float (&sums)[2][kTokens / 4]) {
  constexpr int kPer = kTokens / 4;  // tokens a lane
  const int t8 = (lane & 3) * 8;
  const bool odd_column = (lane & 4) != 0;  // four tokens: this lane's column of B is an odd sub-block's
  const int base[4] = {kFloatBits, kFloatBits, kFloatBits, kFloatBits};
  uint4 head[2] = {*reinterpret_cast<const uint4*>(lo), *reinterpret_cast<const uint4*>(hi)};
  float pr[2][kPer][2] = {}, mr[2][kPer][2] = {};  // [row g / g + 8][token][even / odd sub-blocks]
  const auto chunk = [&](auto index) {
    constexpr int cc = decltype(index)::value;
    const uint2 x = *reinterpret_cast<const uint2*>(lo + 16 + (cc * 32) + t8);
    const uint2 y = *reinterpret_cast<const uint2*>(hi + 16 + (cc * 32) + t8);
    float dot[2][kPer][2];
    float d8[kPer][2], z8[kPer][2];
    if constexpr (kTokens == 8) {
      const uint4 b = *reinterpret_cast<const uint4*>(codes + (c * 256) + (cc * 64));
      const float4 even_scale = *reinterpret_cast<const float4*>(scales + (c * 128) + (cc * 32));
      const float4 odd_scale = *reinterpret_cast<const float4*>(scales + (c * 128) + (cc * 32) + 16);
      int even[4], odd[4];
      MmaOnto(even, x.x & 0x0f0f0f0fu, y.x & 0x0f0f0f0fu, x.y & 0x0f0f0f0fu, y.y & 0x0f0f0f0fu, b.x, b.y, base);
      MmaOnto(odd, x.x & 0xf0f0f0f0u, y.x & 0xf0f0f0f0u, x.y & 0xf0f0f0f0u, y.y & 0xf0f0f0f0u, b.z, b.w, base);
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
          dot[h][j][0] = SumOf(even[(2 * h) + j]);
          dot[h][j][1] = SumOf(odd[(2 * h) + j]);
        }
      d8[0][0] = even_scale.x; d8[kPer - 1][0] = even_scale.y; z8[0][0] = even_scale.z; z8[kPer - 1][0] = even_scale.w;
      d8[0][1] = odd_scale.x; d8[kPer - 1][1] = odd_scale.y; z8[0][1] = odd_scale.z; z8[kPer - 1][1] = odd_scale.w;
    } else {
      const uint2 b = *reinterpret_cast<const uint2*>(codes + (c * 256) + (cc * 64));
      const float4 scale = *reinterpret_cast<const float4*>(scales + (c * 64) + (cc * 16));
      // even sub-block into the even columns, the odd one into the odd
      int both[4];
      MmaOnto(both, x.x & 0x0f0f0f0fu, y.x & 0x0f0f0f0fu, x.y & 0x0f0f0f0fu, y.y & 0x0f0f0f0fu,
              odd_column ? 0u : b.x, odd_column ? 0u : b.y, base);
      MmaOnto(both, x.x & 0xf0f0f0f0u, y.x & 0xf0f0f0f0u, x.y & 0xf0f0f0f0u, y.y & 0xf0f0f0f0u,
              odd_column ? b.x : 0u, odd_column ? b.y : 0u, both);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        dot[h][0][0] = SumOf(both[2 * h]);
        dot[h][0][1] = SumOf(both[(2 * h) + 1]);
      }
      d8[0][0] = scale.x; d8[0][1] = scale.y; z8[0][0] = scale.z; z8[0][1] = scale.w;
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      // the 6-bit scales and minima of sub-blocks 0..3 or 4..7, a byte each
      const uint4 hd = head[h];
      const std::uint32_t sc = cc < 2 ? hd.y & 0x3f3f3f3fu : (hd.w & 0x0f0f0f0fu) | ((hd.y >> 2) & 0x30303030u);
      const std::uint32_t mn = cc < 2 ? hd.z & 0x3f3f3f3fu : ((hd.w >> 4) & 0x0f0f0f0fu) | ((hd.z >> 2) & 0x30303030u);
      constexpr int i = 2 * (cc & 1);
      const float scale[2] = {ByteFloat<i>(sc), ByteFloat<i + 1>(sc)};
      const float minimum[2] = {ByteFloat<i>(mn), ByteFloat<i + 1>(mn)};
#pragma unroll
      for (int j = 0; j < kPer; ++j)
#pragma unroll
        for (int o = 0; o < 2; ++o) {
          pr[h][j][o] = fmaf(d8[j][o] * scale[o], dot[h][j][o], pr[h][j][o]);
          mr[h][j][o] = fmaf(z8[j][o], minimum[o], mr[h][j][o]);
        }
    }
  };
  chunk(Index<0>{});
  chunk(Index<1>{});
  chunk(Index<2>{});
  chunk(Index<3>{});
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const float d = HalfBitsToFloat(head[h].x & 0xffffu), dm = HalfBitsToFloat(head[h].x >> 16);
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      sums[h][j] = fmaf(d, pr[h][j][0] + pr[h][j][1], -(dm * (mr[h][j][0] + mr[h][j][1])));
    }
  }
}

}  // namespace vecq
}  // namespace llmp_b200

#endif  // LLMP_B200_CSRC_VECQ_COLUMNS_CUH_
