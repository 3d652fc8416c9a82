// The unit of the routed batch kernel (vecq_routed.cuh): 16 weight rows x one
// Q4_K super-block x eight activation rows ("tokens"), a warp's work between two waits.
//
//   * The integer products: mma.sync m16n8k32 (u8 x s8 -> s32), one a 32-value sub-block, the
//     rows' 4-bit codes straight out of the staged blocks: lane (g, t) takes bytes 8t..8t+7 of a
//     32-byte chunk of rows g and g + 8, the low nibbles for the chunk's even sub-block, the high
//     ones, left in place as 16 x code, for the odd (1/16, exactly, is on the token's scale).
//     The k slots are a free permutation as long as A and B agree.
//   * The fold: lane (g, t) holds rows g and g + 8 x tokens 2t and 2t + 1 and adds
//     d8 * (sc * dot) and (d8 * sum q) * m, the even and the odd sub-blocks apart (half the
//     roundings in a row).
// The integer ALU takes two cycles a warp instruction on this part, and the fold as the dense
// token-column kernel writes it is mostly its work (conversions, byte extracts, masks) beside idle
// multiply-add pipes.  So what can be goes to them: sc * dot lands in a float by ONE integer
// multiply-add with the bits of 1.5 * 2^23 (|sc * dot| < 2^22; not so for the odd sub-blocks, whose
// dots are 16 times too large) and the minima by one byte permute under 2^23's exponent, each less
// its constant by an exact F32 add; a byte is one permute.  The ALU pipe is then busy 34 % of the
// time and the multiply-add pipes 19 % (a tile's latency, not its issue slots, is what the kernel
// waits for).  (The minima as a BF16 contraction on the tensor core, d8 * sum q in three exact
// pieces: fewer instructions still, but its sums are off by a quarter more.)
#ifndef LLMP_B200_CSRC_VECQ_UNIT_CUH_
#define LLMP_B200_CSRC_VECQ_UNIT_CUH_

#include <cfloat>

#include "vecq_rowmma.cuh"

namespace llmp_b200 {
namespace vecq {

constexpr int kUnitTokens = 8;  // the MMA's columns

// The staged activations of up to eight tokens over `columns` super-block columns:
//   per token: int8, chunk by chunk (a chunk: two sub-blocks): for t = 0..3 bytes 8t..8t+7 of the
//   even sub-block, then of the odd;
//   per pair of tokens: (d8, d8, d8 * sum q, d8 * sum q) a sub-block.
struct TokenActs {
  int columns;
  __host__ __device__ constexpr explicit TokenActs(int c) : columns(c) {}
  // lanes of two tokens read 128 bits at once: 64 bytes modulo 128
  __host__ __device__ constexpr int Pitch() const { return (columns * 256) + 64; }
  // the four pairs' scales are read together: 32 bytes modulo 128
  __host__ __device__ constexpr int PairPitch() const { return (columns * 128) + 32; }
  __host__ __device__ constexpr int Scales() const { return kUnitTokens * Pitch(); }
  __host__ __device__ constexpr int Bytes() const {
    return ((Scales() + (kUnitTokens / 2 * PairPitch())) + 127) / 128 * 128;
  }
};

// One Q8_1 block (sub-block b of the staged columns) of token p.
__device__ __forceinline__ void StageUnitBlock(unsigned char* acts, TokenActs layout, int p, int b,
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
  unsigned char* row = acts + (p * layout.Pitch());
  auto* codes = reinterpret_cast<uint2*>(row + ((b >> 1) * 64) + ((b & 1) * 8));
#pragma unroll
  for (int t = 0; t < 4; ++t) codes[2 * t] = make_uint2(v[2 * t], v[(2 * t) + 1]);
  float* scales = reinterpret_cast<float*>(acts + layout.Scales() + ((p >> 1) * layout.PairPitch())) +
                  (4 * b) + (p & 1);
  scales[0] = (b & 1) != 0 ? d * 0.0625f : d;
  scales[2] = d * static_cast<float>(isum);
}

// An integer below 2^22 in magnitude times another, plus 1.5 * 2^23's bits, as the product's float.
__device__ __forceinline__ float ProductFloat(int a, int b) {
  return __int_as_float((a * b) + 0x4b400000) - 12582912.0f;
}
template <int i>
__device__ __forceinline__ int ByteInt(std::uint32_t w) {
  return static_cast<int>(__byte_perm(w, 0u, 0x4440u | i));
}

// A lane's places in the staged activations; `live` tokens, of which a lane of an absent column
// reads the last one's codes (its results are not stored).
struct UnitLane {
  const unsigned char* codes;
  const unsigned char* scales;
  __device__ __forceinline__ UnitLane(const unsigned char* acts, TokenActs layout, int live, int lane) {
    const int g = lane >> 2, t = lane & 3;
    codes = acts + (min(g, live - 1) * layout.Pitch()) + (16 * t);
    scales = acts + layout.Scales() + (t * layout.PairPitch());
  }
};

// The rounding of a sum or product that is infinite comes out as inf - inf: a number in its place,
// and the infinity it is added to stands.  (One instruction, where a test of the sum is two and a
// register: the two-matrix kernel has none to spare.)
__device__ __forceinline__ float Finite(float rounding) { return fmaxf(rounding, -FLT_MAX); }

// sums[row g / g + 8][token 2t / 2t + 1] += the unit, for `mats` matrices whose blocks of rows g and
// g + 8 start at lo[m] and hi[m]; c: the column among the staged ones.
template <int kMats>
__device__ __forceinline__ void TokenUnit(const unsigned char* const (&lo)[kMats],
                                          const unsigned char* const (&hi)[kMats], const UnitLane& lane,
                                          int t8, int c, float (&sums)[kMats][2][2]) {
  uint4 head[kMats][2];
  // [row g / g + 8][token 2t / 2t + 1][even / odd sub-blocks]
  float pr[kMats][2][2][2], mr[kMats][2][2][2];
#pragma unroll
  for (int m = 0; m < kMats; ++m) {
    head[m][0] = *reinterpret_cast<const uint4*>(lo[m]);
    head[m][1] = *reinterpret_cast<const uint4*>(hi[m]);
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int j = 0; j < 2; ++j) pr[m][h][j][0] = pr[m][h][j][1] = mr[m][h][j][0] = mr[m][h][j][1] = 0.0f;
  }
  // sub-blocks 2cc (low nibbles) and 2cc + 1 (high)
  const auto chunk = [&](auto index) {
    constexpr int cc = decltype(index)::value;
    const uint4 b = *reinterpret_cast<const uint4*>(lane.codes + (c * 256) + (cc * 64));
    const float4 even_scale = *reinterpret_cast<const float4*>(lane.scales + (c * 128) + (cc * 32));
    const float4 odd_scale = *reinterpret_cast<const float4*>(lane.scales + (c * 128) + (cc * 32) + 16);
#pragma unroll
    for (int m = 0; m < kMats; ++m) {
      const uint2 x = *reinterpret_cast<const uint2*>(lo[m] + 16 + (cc * 32) + t8);
      const uint2 y = *reinterpret_cast<const uint2*>(hi[m] + 16 + (cc * 32) + t8);
      int even[4] = {0, 0, 0, 0}, odd[4] = {0, 0, 0, 0};
      MmaU8S8(even, x.x & 0x0f0f0f0fu, y.x & 0x0f0f0f0fu, x.y & 0x0f0f0f0fu, y.y & 0x0f0f0f0fu, b.x, b.y);
      MmaU8S8(odd, x.x & 0xf0f0f0f0u, y.x & 0xf0f0f0f0u, x.y & 0xf0f0f0f0u, y.y & 0xf0f0f0f0u, b.z, b.w);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        // the 6-bit scales and minima of sub-blocks 0..3 or 4..7, a byte each
        const uint4 hd = head[m][h];
        const std::uint32_t sc = cc < 2 ? hd.y & 0x3f3f3f3fu : (hd.w & 0x0f0f0f0fu) | ((hd.y >> 2) & 0x30303030u);
        const std::uint32_t mn = cc < 2 ? hd.z & 0x3f3f3f3fu : ((hd.w >> 4) & 0x0f0f0f0fu) | ((hd.z >> 2) & 0x30303030u);
        constexpr int i = 2 * (cc & 1);
        const int sc0 = ByteInt<i>(sc), sc1 = ByteInt<i + 1>(sc);
        const float mn0 = ByteFloat<i>(mn), mn1 = ByteFloat<i + 1>(mn);
        pr[m][h][0][0] = fmaf(even_scale.x, ProductFloat(even[2 * h], sc0), pr[m][h][0][0]);
        pr[m][h][1][0] = fmaf(even_scale.y, ProductFloat(even[(2 * h) + 1], sc0), pr[m][h][1][0]);
        pr[m][h][0][1] = fmaf(odd_scale.x, static_cast<float>(odd[2 * h] * sc1), pr[m][h][0][1]);
        pr[m][h][1][1] = fmaf(odd_scale.y, static_cast<float>(odd[(2 * h) + 1] * sc1), pr[m][h][1][1]);
        mr[m][h][0][0] = fmaf(even_scale.z, mn0, mr[m][h][0][0]);
        mr[m][h][1][0] = fmaf(even_scale.w, mn0, mr[m][h][1][0]);
        mr[m][h][0][1] = fmaf(odd_scale.z, mn1, mr[m][h][0][1]);
        mr[m][h][1][1] = fmaf(odd_scale.w, mn1, mr[m][h][1][1]);
      }
    }
  };
  chunk(Index<0>{});
  chunk(Index<1>{});
  chunk(Index<2>{});
  chunk(Index<3>{});
#pragma unroll
  for (int m = 0; m < kMats; ++m)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const float d = HalfBitsToFloat(head[m][h].x & 0xffffu), dm = -HalfBitsToFloat(head[m][h].x >> 16);
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        // d * p - dmin * q with one rounding of the two products
        const float p = pr[m][h][j][0] + pr[m][h][j][1], q = mr[m][h][j][0] + mr[m][h][j][1];
        const float main = d * p;
        sums[m][h][j] += fmaf(dm, q, main) + Finite(fmaf(d, p, -main));
      }
    }
}

// The sum of `columns` partial sums `stride` floats apart, in order, with the roundings carried
// along (Knuth's two-sum) and added at the end: the columns' meeting adds one rounding, not one a
// column.  Four loads are in flight together.
__device__ __forceinline__ float SumColumns(const float* at, int columns, int stride) {
  float sum = 0.0f, rest = 0.0f;
  const auto add = [&](float v) {
    const float total = sum + v;
    const float part = total - sum;
    rest += (sum - (total - part)) + (v - part);
    sum = total;
  };
  int w = 0;
  for (; w + 4 <= columns; w += 4) {
    const float a = at[w * stride], b = at[(w + 1) * stride], c = at[(w + 2) * stride], d = at[(w + 3) * stride];
    add(a);
    add(b);
    add(c);
    add(d);
  }
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    if (w + i < columns) add(at[(w + i) * stride]);
  }
  return sum + Finite(rest);
}

}  // namespace vecq
}  // namespace llmp_b200

#endif  // LLMP_B200_CSRC_VECQ_UNIT_CUH_
