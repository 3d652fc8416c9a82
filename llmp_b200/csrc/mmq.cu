// MMQ on B200: the prefill product of Q4_K weights with Q8_1-MMQ activations,
// dense or per routed expert.  Semantics follow the reference's use of GGML's
// mul_mat_q (src/kernels/ggml/mul_mat_q.cu:67-130, 453-462, 551-737; the tile
// loop's shape in-tree at mul_mat_q_glu.cu:93-135; the activation block's
// writer at mul_mat_q_glu.cu:170-218): per 32-value group an exact int32
// product C = sum code * q, then in F32
//     sum += (d * sc)_half * d8 * C;   sum += (-dmin * m)_half * s8
// with d8, s8 the group's FP16 scale and stored input sum.
//
// The int8 contraction runs on tcgen05 (kind::i8, int32 accumulators in TMEM).
// Q4_K's per-group scales forbid accumulating across groups in the tensor
// core, so every group's 128 x 128 x 32 product has to be read out of TMEM and
// folded into F32 register accumulators, and that fold is what bounds the kernel.
// The tensor core, idle for most of it, also forms the group's SCALE products:
// d8 (per token) x (d*sc)_half (per weight row) is a rank-1 FP16 product (kind::f16, K
// 16 of which one is not zero, F32 accumulate: 22 bits, exact), written beside the
// integers, so the fold is two TMEM loads a piece, a conversion a value and one packed
// multiply-add a pair: acc += C * (d8 * d*sc), one rounding.  Every tile has one MMA kind
// and shape between two hand-overs: PTX orders two MMAs in flight only where they share the
// accumulator and the shape.  (So the integers do not accumulate onto the bits of 1.5 * 2^23
// left by a third rank-1 product, which would spare the conversion, two cycles a warp
// instruction: 4096 tokens x 4096 -> 14336 1195 us for 1223, a routed block of 4096 tokens 1238
// for 1304, but nothing says in which order the two kinds would be done, and a commit and a
// wait between them take 1497 and 1513.  The scales by 20 registers a thread, TMEM loads in an
// MMA fragment's layout and four integer buffers: 1595.  With the scales as broadcast
// shared-memory loads, two packed instructions a pair and 16 warps of 32 rows: 139 warp
// instructions and 1,030 cycles a group; 2.4e-7 off the double product where this is 2.1e-7.
// 4096 tokens x 4096 -> 14336: 1.76 ms then, 1.22 now.)
// The MMA's M side (the TMEM lanes) is the TOKENS and its N side (the TMEM columns) the
// weight rows: a thread's results are contiguous in the output.
// The min terms need no integer product: sum over groups of (-dmin*m)_half *
// s8_half is a plain FP16 contraction over K = k / 32, which the tensor core
// takes (kind::f16, F32 accumulate) from two small K-major FP16 tiles: every 64
// groups it takes a TMEM buffer's turn, and the epilogue adds it.
//
// Weights reach the MMA in one of two ways.
//   * SLAB (llmp_b200_q4k_relayout once at load time, or per call into caller
//     scratch): the Q4_K blocks unpacked to what the tensor core reads, int8
//     codes K-major, (d*sc)_half as F32 in [k-step][group][row] tiles, (-dmin*m)
//     half K-major; the producer warp's TMA brings the codes and minima straight into
//     the swizzled tiles.
//   * RAW (no slab, no scratch): two decode warps unpack the Q4_K blocks of a
//     TMA-fed raw stage into the same tiles, k-step by k-step.
//
// One persistent CTA an SM (all of its tensor memory): the next tile's operands and
// first groups are on their way under a tile's write-back.
//
//   warp 0       TMA producer: per k-step the activation int8 tile (128 tokens x
//                128 K bytes) straight out of the [k/128][col] block array through
//                a 3-D tensor map (row pitch 144 B, origin past the 16-byte block
//                header) and, with a slab, the weight tile; per two k-steps the tokens'
//                block headers and the weight rows' scales (raw: their Q4_K blocks) into
//                a raw stage;
//   warp 1       allocates TMEM and issues the MMAs;
//   warps 2-3    the scale tiles (d8; d*sc) and s8 (the min tile) of a k-step; raw mode:
//                also the weight blocks into the int8 tile and -dmin*m;
//   warps 4-11   epilogue: thread = (token, half of the weight rows).
// Rows past the matrix and tokens past the batch are TMA's zero fill.
// Every wait is bounded; a wait that runs out raises the device fault counter.
#include <algorithm>

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "mmq.cuh"
#include "tc.cuh"

namespace llmp_b200 {
namespace {

using Desc = llmp_b200_mmq_desc;

// ------------------------------------------------------------------ quantizer
// block_q8_1_mmq, DS4 layout: 4 x (FP16 d, FP16 sum of the inputs), 128 int8.
// Blocks ordered [k / 128][col].  A warp takes 256 values of k of kCols columns, a lane eight of a
// 32-value group: 16- or 32-byte loads, all columns' on their way together, and neighbouring columns'
// blocks, neighbours in memory, by one warp.  (A thread four values of one column, with a 64-bit
// division each, was bound by its instructions: 28.5 us for 4096 x 4096 BF16 values, 1.8 TB/s.)
// The stored sum's order is four values in order, then parts 4, 2, 1 apart.
// kSlots: column t is quantized once and its blocks go to every column position[t * used + j] >= 0
// (a routed token's rows), where ids_src would have a column's input read and quantized `used` times.
template <bool kBf16>
__device__ __forceinline__ void Load8(const void* __restrict__ x, std::int64_t at, float (&v)[8]) {
  if constexpr (kBf16) {
    const uint4 raw = *reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(x) + at);
    const std::uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      v[2 * i] = __uint_as_float(w[i] << 16);
      v[(2 * i) + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
  } else {
    const float4* from = reinterpret_cast<const float4*>(static_cast<const float*>(x) + at);
    const float4 lo = from[0], hi = from[1];
    v[0] = lo.x; v[1] = lo.y; v[2] = lo.z; v[3] = lo.w;
    v[4] = hi.x; v[5] = hi.y; v[6] = hi.z; v[7] = hi.w;
  }
}

template <bool kBf16, int kCols, bool kSlots>
__global__ void __launch_bounds__(256)
QuantizeMmqKernel(const void* __restrict__ x, std::int64_t row_stride, int k, int cols,
                  const std::int32_t* __restrict__ ids_src, const std::int32_t* __restrict__ position,
                  int used, std::uint8_t* __restrict__ out, unsigned warps) {
  GridLaunchDependents();
  const int lane = static_cast<int>(threadIdx.x) & 31;
  const unsigned chunks = (static_cast<unsigned>(k) + 255u) / 256u;
  const unsigned warp = (blockIdx.x * 8u) + (threadIdx.x >> 5);
  const int at_k = static_cast<int>(((warp % chunks) * 256u) + (static_cast<unsigned>(lane) * 8u));
  const int col0 = static_cast<int>(warp / chunks) * kCols;
  const bool live = warp < warps && at_k < k;
  const std::int64_t out_cols = kSlots ? static_cast<std::int64_t>(cols) * used : cols;
  GridDependencyWait();
  float v[kCols][8];
#pragma unroll
  for (int c = 0; c < kCols; ++c) {
    const int col = min(col0 + c, cols - 1);
    if (live) {
      Load8<kBf16>(x, (static_cast<std::int64_t>(ids_src != nullptr ? ids_src[col] : col) * row_stride) + at_k, v[c]);
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) v[c][i] = 0.0f;
    }
  }
#pragma unroll
  for (int c = 0; c < kCols; ++c) {
    float amax = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(v[c][i]));
    // parts 2j and 2j + 1 of the group's eight (j = lane % 4): parts 4 apart are two lanes apart
    float even = ((v[c][0] + v[c][1]) + v[c][2]) + v[c][3];
    float odd = ((v[c][4] + v[c][5]) + v[c][6]) + v[c][7];
#pragma unroll
    for (int offset = 2; offset > 0; offset >>= 1) {
      amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, offset));
      even = even + __shfl_xor_sync(0xffffffffu, even, offset);
      odd = odd + __shfl_xor_sync(0xffffffffu, odd, offset);
    }
    const float sum = even + odd;
    if (!live || col0 + c >= cols) continue;
    std::uint32_t packed[2] = {0, 0};
    float d = 0.0f;
    if (amax > 0.0f) {
      const float d_inv = 127.0f / amax;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int q = static_cast<int>(roundf(v[c][i] * d_inv));
        packed[i >> 2] |= (static_cast<std::uint32_t>(q) & 0xffu) << (8 * (i & 3));
      }
      d = 1.0f / d_inv;
    }
    const std::uint32_t ds = static_cast<std::uint32_t>(__half_as_ushort(__float2half_rn(d))) |
                             (static_cast<std::uint32_t>(__half_as_ushort(__float2half_rn(sum))) << 16);
    const auto store = [&](std::int64_t col) {
      std::uint8_t* block = out + ((static_cast<std::int64_t>(at_k >> 7) * out_cols) + col) * 144;
      *reinterpret_cast<uint2*>(block + 16 + (at_k & 127)) = make_uint2(packed[0], packed[1]);
      if ((lane & 3) == 0) *reinterpret_cast<std::uint32_t*>(block + ((at_k & 127) >> 3)) = ds;
    };
    if constexpr (kSlots) {
      for (int j = 0; j < used; ++j) {
        const int row = position[(static_cast<std::int64_t>(col0 + c) * used) + j];
        if (row >= 0) store(row);
      }
    } else {
      store(col0 + c);
    }
  }
}

// Four columns a warp where that still fills the chip four times over, else one (203 columns of 2560
// values would be 510 warps of four).
template <bool kBf16, bool kSlots>
int QuantizeMmq(const void* x, std::int64_t row_stride, std::int64_t k, std::int64_t cols,
                const std::int32_t* ids_src, const std::int32_t* position, int used, void* out, void* stream) {
  const std::int64_t chunks = (k + 255) / 256;
  const bool four = ((cols + 3) / 4) * chunks >= static_cast<std::int64_t>(SmCount()) * 32;
  const std::int64_t warps = chunks * (four ? (cols + 3) / 4 : cols);
  if (cols > 0x7fffffffLL || k > 0x7fffffffLL || (warps + 7) / 8 > 0x1fffffffLL) {
    return Reject("mmq.quantize: more blocks than a grid holds");
  }
  const auto kernel = four ? &QuantizeMmqKernel<kBf16, 4, kSlots> : &QuantizeMmqKernel<kBf16, 1, kSlots>;
  const cudaError_t e =
      LaunchPdl(kernel, dim3(static_cast<unsigned>((warps + 7) / 8)), dim3(256), 0, static_cast<cudaStream_t>(stream),
                x, row_stride, static_cast<int>(k), static_cast<int>(cols), ids_src, position, used,
                static_cast<std::uint8_t*>(out), static_cast<unsigned>(warps));
  if (e != cudaSuccess) return Failed(e, "mmq.quantize launch");
  return 0;
}

// ------------------------------------------------------------------ slab
// The weights unpacked for the tensor core (llmp_b200_q4k_relayout).  Per expert:
//   codes  int8  [n][k]                      K-major rows, the MMA's B operand
//   ax     F32   [n / 128 up][k / 128][4][128]   (d * sc)_half of a tile's rows, a
//                                            k-step's four groups: 2 KB contiguous
//   mw     FP16  [n][G]                      (-dmin * m)_half, K-major; G = k / 32
//                                            rounded up to 64 (zero padding)
struct Slab {
  std::size_t codes, ax, mw, total;
  int row_tiles, ksteps, gpad;
};
Slab SlabOf(int n, int k, int experts) {
  Slab s;
  s.row_tiles = (n + 127) / 128;
  s.ksteps = k / 128;
  s.gpad = ((k / 32) + 63) / 64 * 64;
  const auto up = [](std::size_t v) { return (v + 255) / 256 * 256; };
  s.codes = 0;
  s.ax = up(static_cast<std::size_t>(experts) * n * k);
  s.mw = s.ax + up(static_cast<std::size_t>(experts) * s.row_tiles * s.ksteps * 512 * 4);
  s.total = s.mw + up(static_cast<std::size_t>(experts) * n * s.gpad * 2);
  return s;
}

__device__ __forceinline__ void ScaleAndMin(std::uint32_t s0, std::uint32_t s1, std::uint32_t s2,
                                            int g, int* sc, int* mn) {
  // 6-bit fields: groups 0..3 in the low six bits of bytes 0..3 (scales) and 4..7
  // (minima); groups 4..7 as the nibbles of bytes 8..11 with their top two bits in
  // bits 6..7 of bytes 0..3 / 4..7.
  const int gl = g & 3;
  if (g < 4) {
    *sc = static_cast<int>((s0 >> (8 * gl)) & 63u);
    *mn = static_cast<int>((s1 >> (8 * gl)) & 63u);
  } else {
    *sc = static_cast<int>(((s2 >> (8 * gl)) & 15u) | (((s0 >> ((8 * gl) + 6)) & 3u) << 4));
    *mn = static_cast<int>(((s2 >> ((8 * gl) + 4)) & 15u) | (((s1 >> ((8 * gl) + 6)) & 3u) << 4));
  }
}

// A warp takes 32 consecutive rows of one super-block column: lane = row, so the
// scale tiles are written 128 bytes a warp.
__global__ void __launch_bounds__(256)
RelayoutQ4KKernel(const std::uint8_t* __restrict__ w, int n, int k, std::int64_t stride_row,
                  std::int64_t stride_expert, int experts, std::uint8_t* __restrict__ slab,
                  const Slab layout, int glu_inter) {
  GridLaunchDependents();
  GridDependencyWait();  // the slab may still be read by the product queued before
  const int lane = static_cast<int>(threadIdx.x) & 31;
  const int sbs = k / 256;
  const int row_groups = layout.row_tiles * 4;  // 32-row groups an expert, padding included
  const std::int64_t item = (static_cast<std::int64_t>(blockIdx.x) * 8) + (threadIdx.x >> 5);
  if (item >= static_cast<std::int64_t>(experts) * row_groups * sbs) return;
  const int sb = static_cast<int>(item % sbs);
  const int rg = static_cast<int>((item / sbs) % row_groups);
  const int e = static_cast<int>(item / (static_cast<std::int64_t>(sbs) * row_groups));
  const int row = (rg * 32) + lane;
  const bool live = row < n;
  uint4 head = make_uint4(0, 0, 0, 0), q[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) q[i] = make_uint4(0, 0, 0, 0);
  // For the GLU write-back the slab's rows interleave the gate and up rows (the source holds
  // glu_inter gate rows, then as many up rows): slab rows 32g .. 32g + 15 are gate rows
  // 16g .. 16g + 15 and slab rows 32g + 16 .. 32g + 31 the up rows of the same outputs, so an
  // epilogue thread's 32 rows are 16 (gate, up) pairs.
  int from = row;
  if (glu_inter > 0) from = (lane < 16 ? 0 : glu_inter) + (rg * 16) + (lane & 15);
  if (live) {
    const auto* src = reinterpret_cast<const uint4*>(
        w + ((static_cast<std::int64_t>(e) * stride_expert + static_cast<std::int64_t>(from) * stride_row + sb) * 144));
    head = LoadStream16(src);
#pragma unroll
    for (int i = 0; i < 8; ++i) q[i] = LoadStream16(src + 1 + i);
  }
  const __half d = __ushort_as_half(static_cast<unsigned short>(head.x & 0xffffu));
  const __half dmin = __hneg(__ushort_as_half(static_cast<unsigned short>(head.x >> 16)));
  float* ax = reinterpret_cast<float*>(slab + layout.ax) +
              ((static_cast<std::int64_t>(e) * layout.row_tiles + (row >> 7)) * layout.ksteps * 512);
  std::uint32_t mins[4];
#pragma unroll
  for (int g = 0; g < 8; ++g) {
    int scv, mnv;
    ScaleAndMin(head.y, head.z, head.w, g, &scv, &mnv);
    // the half-precision products of GGML's tile loader
    ax[((((2 * sb) + (g >> 2)) * 4 + (g & 3)) * 128) + (row & 127)] =
        live ? __half2float(__hmul(d, __int2half_rn(scv))) : 0.0f;
    const std::uint32_t bits = live ? __half_as_ushort(__hmul(dmin, __int2half_rn(mnv))) : 0u;
    if ((g & 1) == 0) {
      mins[g >> 1] = bits;
    } else {
      mins[g >> 1] |= bits << 16;
    }
  }
  if (!live) return;
  auto* codes = reinterpret_cast<uint4*>(
      slab + layout.codes + ((static_cast<std::int64_t>(e) * n + row) * k) + (static_cast<std::int64_t>(sb) * 256));
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const uint4 a = q[2 * c], b = q[(2 * c) + 1];
    codes[(4 * c) + 0] = make_uint4(a.x & 0x0f0f0f0fu, a.y & 0x0f0f0f0fu, a.z & 0x0f0f0f0fu, a.w & 0x0f0f0f0fu);
    codes[(4 * c) + 1] = make_uint4(b.x & 0x0f0f0f0fu, b.y & 0x0f0f0f0fu, b.z & 0x0f0f0f0fu, b.w & 0x0f0f0f0fu);
    codes[(4 * c) + 2] = make_uint4((a.x >> 4) & 0x0f0f0f0fu, (a.y >> 4) & 0x0f0f0f0fu,
                                    (a.z >> 4) & 0x0f0f0f0fu, (a.w >> 4) & 0x0f0f0f0fu);
    codes[(4 * c) + 3] = make_uint4((b.x >> 4) & 0x0f0f0f0fu, (b.y >> 4) & 0x0f0f0f0fu,
                                    (b.z >> 4) & 0x0f0f0f0fu, (b.w >> 4) & 0x0f0f0f0fu);
  }
  auto* mw = reinterpret_cast<uint4*>(slab + layout.mw +
                                      ((static_cast<std::int64_t>(e) * n + row) * layout.gpad * 2));
  mw[sb] = make_uint4(mins[0], mins[1], mins[2], mins[3]);
  if (sb == sbs - 1) {
    for (int pad = sbs; pad < layout.gpad / 8; ++pad) mw[pad] = make_uint4(0, 0, 0, 0);
  }
}

// ------------------------------------------------------------------ GEMM
constexpr int kTileCols = 128;  // tokens: the MMA's M, one TMEM lane each
// Weight rows: the MMA's N, one TMEM column each.  128, or 64 where the tiles of 128 leave SMs idle
// (LaunchMmq): the same sums in the same order.
constexpr int kTileRows = 128;
constexpr int kBK = 128;        // K bytes a stage: four 32-value groups
constexpr int kStages = 3;
// A TMEM buffer holds a group's integer tile and, beside it, its scale tile; two of them are all
// 512 columns, so the min terms' sum takes a buffer's turn instead of columns of its own.
template <int kRows>
constexpr int kBuffers = 256 / kRows;
constexpr int kMaxBuffers = 4;
template <int kRows>
constexpr int kBufferColumns = 2 * kRows;
constexpr int kWBytes = kTileRows * kBK, kYBytes = kTileCols * kBK;
// The scale tile's operands, one pair a group: K 16 of which only k = 0 is not zero.  K-major
// without swizzle: 8 rows x 16 bytes (k = 0..7) a core matrix, the groups of 8 rows 128 bytes
// apart; k = 8..15 of every operand is one shared tile of zeros, reached by the leading offset.
constexpr int kScaleTileBytes = 128 * 16;
constexpr int kStageScaleBytes = 4 * kScaleTileBytes;  // [group]
constexpr int kStageBytes = kWBytes + kYBytes + (2 * kStageScaleBytes);
// The min terms' operands: FP16 [128 rows or tokens][64 groups] K-major, 128-byte
// swizzled like the int8 tiles; one tile holds 16 k-steps.  With a slab two tiles alternate,
// raw blocks leave room for one.
constexpr int kMinTileBytes = 128 * 128;
constexpr int kMinSteps = 16;  // k-steps a tile of min operands covers
template <bool kSlab>
constexpr int kMinTiles = kSlab ? 2 : 1;
// Raw stages: what TMA brings for one super-block column (two k-steps): the 128 weight rows'
// Q4_K blocks, or with a slab the rows' scales of both k-steps; then the 128 tokens' block
// headers of both.
constexpr int kRawStages = 2;
constexpr int kAxBytes = 4 * 128 * 4;  // a k-step's d * sc in a slab
template <bool kSlab>
constexpr int kRawWBytes = kSlab ? 2 * kAxBytes : 128 * 144;
constexpr int kRawHBytes = 128 * 16;
template <bool kSlab>
constexpr int kRawBytes = kRawWBytes<kSlab> + (2 * kRawHBytes);
constexpr int kMmaWarp = 1;
constexpr int kFirstDecodeWarp = 2;
constexpr int kDecodeWarps = 2;  // a thread takes two weight rows and two tokens
static_assert(kTileRows == kTileCols, "a row and a token an item");
constexpr int kFirstEpilogueWarp = kFirstDecodeWarp + kDecodeWarps;
// Eight epilogue warps of 64 weight rows a thread rather than 16 of 32: twelve warps leave 168
// registers a thread, which hold the 64 sums and two 16-row pieces, so a piece's loads run under
// the fold of the one before.
constexpr int kEpilogueWarps = 8;
constexpr int kThreads = (kFirstEpilogueWarp + kEpilogueWarps) * 32;
template <int kRows>
constexpr int kEpilogueRows = kRows / (kEpilogueWarps / 4);  // weight rows a thread
static_assert(kEpilogueRows<kTileRows> == 64, "two 32-row groups a thread");
template <bool kSlab>
constexpr int kSmem = (kStages * kStageBytes) + (2 * kMinTiles<kSlab> * kMinTileBytes) +
                      (kRawStages * kRawBytes<kSlab>) + kScaleTileBytes + 512;
static_assert(kSmem<true> <= 232448 && kSmem<false> <= 232448, "a CTA's shared memory");

// Two F32 lanes in one 64-bit register: sm_100's packed F32 arithmetic does two
// roundings-to-nearest per instruction, the same results as two scalar ones.
__device__ __forceinline__ std::uint64_t Pack2(float lo, float hi) {
  std::uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void Unpack2(std::uint64_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ std::uint64_t Add2(std::uint64_t a, std::uint64_t b) {
  std::uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ std::uint64_t Fma2(std::uint64_t a, std::uint64_t b, std::uint64_t c) {
  std::uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

struct Shared {
  std::uint64_t y_full[kStages];   // the stage's TMA bytes have landed
  std::uint64_t w_full[kStages];   // the decode warps have written their part
  std::uint64_t empty[kStages];    // the tensor core has read the stage
  std::uint64_t tmem_full[kMaxBuffers];
  std::uint64_t tmem_empty[kMaxBuffers];
  std::uint64_t raw_full[kRawStages];
  std::uint64_t raw_empty[kRawStages];
  std::uint64_t minw_full[2];  // slab mode: a tile of weight min operands has landed
  std::uint64_t min_free[2];   // the tensor core has read a tile of min operands
  std::uint32_t tmem_base;
  std::uint32_t abort;
};

struct Params {
  Desc a;
  const std::int32_t* worklist;
  unsigned int* faults;
  const float* ax;       // slab: the scale tiles
  int ax_ksteps;         // k-steps a row tile's scales span
  int ax_row_tiles;
  int col_tiles;         // of an expert, or the worklist's capacity
  std::int32_t* sums;    // verification: the int32 group sums [col][row][k / 32]
  // GLU write-back (slab with interleaved gate / up rows): the GLU of every (gate, up) pair,
  // requantized to Q8_1-MMQ blocks [nrows / 2 / 128][ncols], instead of the F32 output.
  std::uint8_t* glu_out;
  int glu;
  float limit;
};

// K-major operand without swizzle: 8-row core matrices 128 bytes apart, the second half of the
// K 16 in the tile at `zeros`.
__device__ __forceinline__ std::uint64_t ScaleDesc(const unsigned char* tile,
                                                   const unsigned char* zeros) {
  const std::uint32_t lbo = (tc::Smem(zeros) - tc::Smem(tile)) >> 4;
  return tc::SmemDesc(tile, false, 128) | (static_cast<std::uint64_t>(lbo & 0x3fffu) << 16);
}

// Both loads of a 16-row piece: the registers of the integers and of the scales are usable only
// after this.
__device__ __forceinline__ void PieceWait(std::uint32_t (&c)[16], std::uint32_t (&s)[16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]), "+r"(c[4]), "+r"(c[5]), "+r"(c[6]),
                 "+r"(c[7]), "+r"(c[8]), "+r"(c[9]), "+r"(c[10]), "+r"(c[11]), "+r"(c[12]),
                 "+r"(c[13]), "+r"(c[14]), "+r"(c[15]), "+r"(s[0]), "+r"(s[1]), "+r"(s[2]),
                 "+r"(s[3]), "+r"(s[4]), "+r"(s[5]), "+r"(s[6]), "+r"(s[7]), "+r"(s[8]), "+r"(s[9]),
                 "+r"(s[10]), "+r"(s[11]), "+r"(s[12]), "+r"(s[13]), "+r"(s[14]), "+r"(s[15])
               :
               : "memory");
}

template <bool kSlab, bool kSums, int kRows>
__global__ void __launch_bounds__(kThreads, 1)
MmqQ4KKernel(const __grid_constant__ CUtensorMap map_y, const __grid_constant__ CUtensorMap map_w,
             const __grid_constant__ CUtensorMap map_h, const __grid_constant__ CUtensorMap map_mw,
             const __grid_constant__ Params p) {
  const Desc& a = p.a;
  constexpr int kMins = kMinTiles<kSlab>;
  extern __shared__ __align__(1024) unsigned char smem[];  // the swizzle's period
  unsigned char* w_tiles = smem;
  unsigned char* y_tiles = w_tiles + (kStages * kWBytes);
  unsigned char* min_w = y_tiles + (kStages * kYBytes);    // [kMins] tiles: (-dmin * m) per weight row
  unsigned char* min_y = min_w + (kMins * kMinTileBytes);  // [kMins] tiles: s8 per token
  unsigned char* scale_w = min_y + (kMins * kMinTileBytes);            // [kStages][group] d * sc
  unsigned char* scale_y = scale_w + (kStages * kStageScaleBytes);     // [kStages][group] d8
  unsigned char* zeros = scale_y + (kStages * kStageScaleBytes);
  unsigned char* raw = zeros + kScaleTileBytes;                        // [kRawStages] raw stages
  Shared* sh = reinterpret_cast<Shared*>(raw + (kRawStages * kRawBytes<kSlab>));

  // (the shuffles tell the compiler that these are the warp's: tensor-memory addresses then live in
  // uniform registers)
  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x) >> 5, 0);
  const int lane = static_cast<int>(threadIdx.x) & 31;
  const int ksteps = a.k / kBK;
  if ((tc::Smem(smem) & 1023u) != 0) {  // uniform: the tiles' layout needs it
    if (threadIdx.x == 0) atomicAdd(p.faults, 1u);
    return;
  }

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      tc::MbarInit(&sh->y_full[s], 1);
      tc::MbarInit(&sh->w_full[s], kDecodeWarps);
      tc::MbarInit(&sh->empty[s], 1);
    }
    for (int b = 0; b < kBuffers<kRows>; ++b) {
      tc::MbarInit(&sh->tmem_full[b], 1);
      tc::MbarInit(&sh->tmem_empty[b], kEpilogueWarps);
    }
    for (int r = 0; r < kRawStages; ++r) {
      tc::MbarInit(&sh->raw_full[r], 1);
      tc::MbarInit(&sh->raw_empty[r], kDecodeWarps);
    }
    for (int t = 0; t < 2; ++t) {
      tc::MbarInit(&sh->minw_full[t], 1);
      tc::MbarInit(&sh->min_free[t], 1);
    }
    sh->abort = 0;
    tc::MbarInitFence();
  }
  if (threadIdx.x < kScaleTileBytes / 16) {
    reinterpret_cast<uint4*>(zeros)[threadIdx.x] = make_uint4(0u, 0u, 0u, 0u);
    tc::FenceProxyAsync();
  }
  if (warp == kMmaWarp) {
    tc::TmemAlloc(&sh->tmem_base, 512);
    tc::TmemRelinquish();
  }
  tc::TcFenceBefore();
  __syncthreads();
  tc::TcFenceAfter();
  // All of the above runs beside the tail of the kernel before (the quantizer, the route, the
  // relayout: everything below may be theirs).
  GridLaunchDependents();
  GridDependencyWait();

  // A CTA takes tiles blockIdx.x, + gridDim.x, ...: weight rows [row0, row0 + 128) of an expert
  // against sorted columns [col0, col0 + 128) of that expert's range, row tiles fastest.  With a
  // worklist (built on the device from the expert bounds) column tile y names entry y: {expert,
  // first column}; entry 0 holds the entry count.
  const int row_tiles = (a.nrows + kRows - 1) / kRows;
  const int col_tiles = p.worklist != nullptr ? min(p.worklist[0], p.col_tiles) : p.col_tiles;
  const std::int64_t tiles = static_cast<std::int64_t>(row_tiles) * col_tiles *
                             (p.worklist == nullptr && a.expert_bounds != nullptr ? a.experts : 1);
  struct Tile {
    int expert, row_tile, col0, c_end;
  };
  const auto tile_at = [&](std::int64_t i) {
    Tile tile;
    tile.row_tile = static_cast<int>(i % row_tiles);
    const std::int64_t rest = i / row_tiles;
    if (p.worklist != nullptr) {
      tile.expert = p.worklist[1 + (2 * rest)];
      tile.col0 = p.worklist[2 + (2 * rest)];
    } else {
      tile.expert = static_cast<int>(rest / col_tiles);
      tile.col0 = (a.expert_bounds != nullptr ? a.expert_bounds[tile.expert] : 0) +
                  (static_cast<int>(rest % col_tiles) * kTileCols);
    }
    tile.c_end = a.expert_bounds != nullptr ? a.expert_bounds[tile.expert + 1] : a.ncols;
    return tile;  // nothing to do, for every role alike, when col0 >= c_end
  };

  const std::uint32_t tmem = __shfl_sync(0xffffffffu, sh->tmem_base, 0);
  volatile std::uint32_t* abort_flag = &sh->abort;
  auto give_up = [&]() {
    *abort_flag = 1;
    atomicAdd(p.faults, 1u);
  };

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    if (lane == 0) {
      tc::PrefetchMap(&map_y);
      tc::PrefetchMap(&map_w);
      tc::PrefetchMap(&map_h);
      if constexpr (kSlab) tc::PrefetchMap(&map_mw);
      std::uint32_t it = 0, column = 0, mins = 0;  // k-steps, super-block columns, min tiles so far
      bool ok = true;
      for (std::int64_t i = blockIdx.x; i < tiles && ok && !*abort_flag; i += gridDim.x) {
        const Tile tile = tile_at(i);
        if (tile.col0 >= tile.c_end) continue;
        const int expert = tile.expert, col0 = tile.col0, row0 = tile.row_tile * kRows;
        for (int ks = 0; ks < ksteps; ++ks, ++it) {
          if ((ks & 1) == 0) {
            // One super-block column (k-steps ks, ks + 1): the tokens' block headers and the
            // weight rows' scales (or, raw, their blocks), for the decode warps.
            const int rs = static_cast<int>(column % kRawStages);
            ok = tc::MbarWaitSleep(&sh->raw_empty[rs], ((column / kRawStages) & 1) ^ 1, 128);
            if (!ok) {
              give_up();
              break;
            }
            unsigned char* stage = raw + (rs * kRawBytes<kSlab>);
            tc::MbarExpectTx(&sh->raw_full[rs], kSlab ? kRawBytes<kSlab> : kRawBytes<kSlab> - ((kTileRows - kRows) * 144));
            if constexpr (kSlab) {
              // k is a multiple of 256: the two k-steps' tiles are 4 KB in a row
              const float* src = p.ax + ((((static_cast<std::int64_t>(expert) * p.ax_row_tiles) +
                                           (tile.row_tile * kRows / kTileRows)) * p.ax_ksteps + ks) * 512);
              tc::BulkLoad(stage, src, 2 * kAxBytes, &sh->raw_full[rs]);
            } else {
              asm volatile(
                  "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
                  " [%0], [%1, {%3, %4, %5}], [%2];"
                  ::"r"(tc::Smem(stage)), "l"(&map_w), "r"(tc::Smem(&sh->raw_full[rs])),
                    "r"((ks >> 1) * 144), "r"(row0), "r"(expert)
                  : "memory");
            }
            asm volatile(
                "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
                " [%0], [%1, {%3, %4, %5}], [%2];"
                ::"r"(tc::Smem(stage + kRawWBytes<kSlab>)), "l"(&map_h),
                  "r"(tc::Smem(&sh->raw_full[rs])), "r"(0), "r"(col0), "r"(ks)
                : "memory");
            ++column;
          }
          if constexpr (kSlab) {
            // Every 16 k-steps a tile of the weight rows' min operands.
            if (ks % kMinSteps == 0) {
              const int mt = static_cast<int>(mins % kMins);
              if (mins >= kMins) ok = tc::MbarWaitSleep(&sh->min_free[mt], ((mins / kMins) - 1) & 1, 128);
              if (!ok) {
                give_up();
                break;
              }
              ++mins;
              tc::MbarExpectTx(&sh->minw_full[mt], kRows * 128);
              asm volatile(
                  "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
                  " [%0], [%1, {%3, %4, %5}], [%2];"
                  ::"r"(tc::Smem(min_w + (mt * kMinTileBytes))), "l"(&map_mw),
                    "r"(tc::Smem(&sh->minw_full[mt])), "r"((ks / kMinSteps) * 128), "r"(row0),
                    "r"(expert)
                  : "memory");
            }
          }
          const int s = static_cast<int>(it % kStages);
          ok = tc::MbarWaitSleep(&sh->empty[s], ((it / kStages) & 1) ^ 1, 64);
          if (!ok) {
            give_up();
            break;
          }
          tc::MbarExpectTx(&sh->y_full[s], kSlab ? kYBytes + (kRows * kBK) : kYBytes);
          asm volatile(
              "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
              " [%0], [%1, {%3, %4, %5}], [%2];"
              ::"r"(tc::Smem(y_tiles + (s * kYBytes))), "l"(&map_y), "r"(tc::Smem(&sh->y_full[s])),
                "r"(0), "r"(col0), "r"(ks)
              : "memory");
          if constexpr (kSlab) {
            asm volatile(
                "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
                " [%0], [%1, {%3, %4, %5}], [%2];"
                ::"r"(tc::Smem(w_tiles + (s * kWBytes))), "l"(&map_w), "r"(tc::Smem(&sh->y_full[s])),
                  "r"(ks * kBK), "r"(row0), "r"(expert)
                : "memory");
          }
        }
      }
    }
  } else if (warp >= kFirstDecodeWarp && warp < kFirstEpilogueWarp) {
    // ------------------------------------------------------------ decode
    // A thread prepares weight rows and tokens t0 and t0 + 64 of every k-step.  Rows past the
    // matrix and tokens past the batch arrive as zero blocks (TMA's fill): zero scales, zero
    // codes, nothing stored for them.
    const int t0 = static_cast<int>(threadIdx.x) - (kFirstDecodeWarp * 32);
    std::uint32_t it = 0, column = 0, mins = 0;
    bool ok = true;
    for (std::int64_t i = blockIdx.x; i < tiles && ok && !*abort_flag; i += gridDim.x) {
      const Tile tile = tile_at(i);
      if (tile.col0 >= tile.c_end) continue;
      for (int ks = 0; ks < ksteps; ++ks, ++it) {
        const int s = static_cast<int>(it % kStages);
        const int half = ks & 1;
        const int rs = static_cast<int>(column % kRawStages);
        const int mt = static_cast<int>(mins % kMins);  // the tile of min operands this k-step writes into
        if (lane == 0) {
          if (half == 0) ok = tc::MbarWait(&sh->raw_full[rs], (column / kRawStages) & 1);
          ok = ok && tc::MbarWait(&sh->empty[s], ((it / kStages) & 1) ^ 1);
          // ... and the tensor core is done with the min tile's contents of kMins tiles ago
          if (mins >= kMins && ks % kMinSteps == 0) {
            ok = ok && tc::MbarWait(&sh->min_free[mt], ((mins / kMins) - 1) & 1);
          }
        }
        ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
        if (!ok) {
          if (lane == 0) give_up();
          break;
        }
        const unsigned char* stage = raw + (rs * kRawBytes<kSlab>);
        const int kk = ks % kMinSteps;
        // a slab's scales come for 128 rows
        const int ax_row = kSlab ? (tile.row_tile * kRows) % kTileRows : 0;
#pragma unroll  // the rows of a thread are independent: their latencies overlap
        for (int t = t0; t < kTileRows; t += kDecodeWarps * 32) {
          const int row_at = ((t >> 3) * 128) + ((t & 7) * 16);  // row t of a scale tile
          unsigned char* sw = scale_w + (s * kStageScaleBytes) + row_at;
          unsigned char* sy = scale_y + (s * kStageScaleBytes) + row_at;
          // Row t of a min tile, the four halves of this k-step: byte (ks % 16) * 8 of
          // the 128-byte row, 16-byte chunks swizzled like the int8 tiles.
          const int at = ((t >> 3) * 1024) + ((t & 7) * 128) + ((((kk >> 1) ^ (t & 7))) * 16) +
                         ((kk & 1) * 8);
          if (t >= kRows) {
            // (a tile of 64 rows: the second half of the tokens only)
          } else if constexpr (kSlab) {
            // (d * sc)_half comes widened to F32: back to half precision, exactly.
            const float* ax = reinterpret_cast<const float*>(stage + (half * kAxBytes)) + ax_row + t;
#pragma unroll
            for (int gl = 0; gl < 4; ++gl) {
              *reinterpret_cast<uint4*>(sw + (gl * kScaleTileBytes)) =
                  make_uint4(__half_as_ushort(__float2half_rn(ax[gl * 128])), 0u, 0u, 0u);
            }
          } else {
            const unsigned char* sb = stage + (t * 144);
            const uint4 head = *reinterpret_cast<const uint4*>(sb);
            uint4 q[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              q[i] = *reinterpret_cast<const uint4*>(sb + 16 + (half * 64) + (i * 16));
            }
            // int8 codes into the swizzled K-major tile: row t, 16-byte chunk j at j ^ (t % 8)
            unsigned char* wt = w_tiles + (s * kWBytes) + ((t >> 3) * 1024) + ((t & 7) * 128);
#pragma unroll
            for (int cc = 0; cc < 2; ++cc) {
              const uint4 lo0 = make_uint4(q[2 * cc].x & 0x0f0f0f0fu, q[2 * cc].y & 0x0f0f0f0fu,
                                           q[2 * cc].z & 0x0f0f0f0fu, q[2 * cc].w & 0x0f0f0f0fu);
              const uint4 lo1 = make_uint4(q[2 * cc + 1].x & 0x0f0f0f0fu, q[2 * cc + 1].y & 0x0f0f0f0fu,
                                           q[2 * cc + 1].z & 0x0f0f0f0fu, q[2 * cc + 1].w & 0x0f0f0f0fu);
              const uint4 hi0 = make_uint4((q[2 * cc].x >> 4) & 0x0f0f0f0fu, (q[2 * cc].y >> 4) & 0x0f0f0f0fu,
                                           (q[2 * cc].z >> 4) & 0x0f0f0f0fu, (q[2 * cc].w >> 4) & 0x0f0f0f0fu);
              const uint4 hi1 = make_uint4((q[2 * cc + 1].x >> 4) & 0x0f0f0f0fu, (q[2 * cc + 1].y >> 4) & 0x0f0f0f0fu,
                                           (q[2 * cc + 1].z >> 4) & 0x0f0f0f0fu, (q[2 * cc + 1].w >> 4) & 0x0f0f0f0fu);
              const int j = cc * 4;  // groups 2cc (chunks j, j+1) and 2cc+1 (chunks j+2, j+3)
              *reinterpret_cast<uint4*>(wt + (((j + 0) ^ (t & 7)) * 16)) = lo0;
              *reinterpret_cast<uint4*>(wt + (((j + 1) ^ (t & 7)) * 16)) = lo1;
              *reinterpret_cast<uint4*>(wt + (((j + 2) ^ (t & 7)) * 16)) = hi0;
              *reinterpret_cast<uint4*>(wt + (((j + 3) ^ (t & 7)) * 16)) = hi1;
            }
            // The four groups' half products (d * sc, -dmin * m): GGML's tile loader
            // multiplies in half precision.
            const __half d = __ushort_as_half(static_cast<unsigned short>(head.x & 0xffffu));
            const __half dmin = __hneg(__ushort_as_half(static_cast<unsigned short>(head.x >> 16)));
            std::uint32_t mins[4];
#pragma unroll
            for (int gl = 0; gl < 4; ++gl) {
              int scv, mnv;
              ScaleAndMin(head.y, head.z, head.w, (half * 4) + gl, &scv, &mnv);
              *reinterpret_cast<uint4*>(sw + (gl * kScaleTileBytes)) =
                  make_uint4(__half_as_ushort(__hmul(d, __int2half_rn(scv))), 0u, 0u, 0u);
              mins[gl] = __half_as_ushort(__hmul(dmin, __int2half_rn(mnv)));
            }
            *reinterpret_cast<uint2*>(min_w + (mt * kMinTileBytes) + at) =
                make_uint2(mins[0] | (mins[1] << 16), mins[2] | (mins[3] << 16));
          }
          // The token's header of this k-step: four (d8, s8) pairs.
          const uint4 ds = *reinterpret_cast<const uint4*>(stage + kRawWBytes<kSlab> +
                                                           (half * kRawHBytes) + (t * 16));
          const std::uint32_t dsw[4] = {ds.x, ds.y, ds.z, ds.w};
#pragma unroll
          for (int gl = 0; gl < 4; ++gl) {
            *reinterpret_cast<uint4*>(sy + (gl * kScaleTileBytes)) = make_uint4(dsw[gl] & 0xffffu, 0u, 0u, 0u);
          }
          *reinterpret_cast<uint2*>(min_y + (mt * kMinTileBytes) + at) =
              make_uint2((dsw[0] >> 16) | (dsw[1] & 0xffff0000u), (dsw[2] >> 16) | (dsw[3] & 0xffff0000u));
          // The last FP16 MMA of the min terms reads 16 groups: zero what the k range leaves unwritten.
          if (ks == ksteps - 1) {
            for (int pad = ks + 1; pad % 4 != 0; ++pad) {
              const int pk = pad % kMinSteps;
              const int pat = ((t >> 3) * 1024) + ((t & 7) * 128) + ((((pk >> 1) ^ (t & 7))) * 16) +
                              ((pk & 1) * 8);
              if (!kSlab && t < kRows) {
                *reinterpret_cast<uint2*>(min_w + (mt * kMinTileBytes) + pat) = make_uint2(0u, 0u);
              }
              *reinterpret_cast<uint2*>(min_y + (mt * kMinTileBytes) + pat) = make_uint2(0u, 0u);
            }
          }
        }
        tc::FenceProxyAsync();  // generic-proxy writes, read by the tensor core's proxy
        __syncwarp();
        if (lane == 0) {
          if (half == 1) tc::MbarArrive(&sh->raw_empty[rs]);  // the raw stage is read
          tc::MbarArrive(&sh->w_full[s]);
        }
        if (half == 1) ++column;
        if (ks % kMinSteps == kMinSteps - 1 || ks == ksteps - 1) ++mins;
      }
    }
  } else if (warp == kMmaWarp) {
    // ------------------------------------------------------------ MMA issuer
    // The whole warp walks the loop and one elected lane issues: from inside a one-lane branch
    // every MMA and commit held the thread 60-70 cycles.
    const bool elected = tc::ElectOne();
    // A (M, the TMEM lanes): tokens, signed int8.  B (N, the TMEM columns): weight
    // rows, unsigned codes.
    const std::uint32_t idesc = tc::IdescI8(kTileCols, kRows, true, false);
    const std::uint32_t fdesc = tc::IdescF16(kTileCols, kRows);
    std::uint32_t turn = 0, it = 0, mins = 0;  // turn: of the TMEM buffers
    bool ok = true;
    for (std::int64_t i = blockIdx.x; i < tiles && ok && !*abort_flag; i += gridDim.x) {
      const Tile tile = tile_at(i);
      if (tile.col0 >= tile.c_end) continue;
      for (int ks = 0; ks < ksteps; ++ks, ++it) {
        const int s = static_cast<int>(it % kStages);
        ok = tc::MbarWait(&sh->w_full[s], (it / kStages) & 1) &&
             tc::MbarWait(&sh->y_full[s], (it / kStages) & 1);
        if (!__all_sync(0xffffffffu, ok)) {
          ok = false;
          break;
        }
        tc::TcFenceAfter();
        const std::uint64_t wdesc = tc::SmemDesc(w_tiles + (s * kWBytes), true, 1024);
        const std::uint64_t ydesc = tc::SmemDesc(y_tiles + (s * kYBytes), true, 1024);
        const unsigned char* sw = scale_w + (s * kStageScaleBytes);
        const unsigned char* sy = scale_y + (s * kStageScaleBytes);
#pragma unroll
        for (int gl = 0; gl < 4; ++gl, ++turn) {
          const int b = static_cast<int>(turn % kBuffers<kRows>);
          const std::uint64_t swd = ScaleDesc(sw + (gl * kScaleTileBytes), zeros);
          const std::uint64_t syd = ScaleDesc(sy + (gl * kScaleTileBytes), zeros);
          ok = tc::MbarWait(&sh->tmem_empty[b], ((turn / kBuffers<kRows>) & 1u) ^ 1u);
          if (!__all_sync(0xffffffffu, ok)) {
            ok = false;
            break;
          }
          tc::TcFenceAfter();
          if (elected) {
            const std::uint32_t d = tmem + (b * kBufferColumns<kRows>);
            tc::MmaI8(d, ydesc + (gl * 2), wdesc + (gl * 2), idesc, false);
            tc::MmaF16(d + kRows, syd, swd, fdesc, false);
            tc::TcCommit(&sh->tmem_full[b]);
            if (gl == 3) tc::TcCommit(&sh->empty[s]);
          }
        }
        if (!ok) break;
        // Every 16 k-steps, and at the end, the min terms of the tile: up to four FP16 MMAs (K 16
        // each, the operands of four k-steps) into the next buffer.
        if (ks % kMinSteps == kMinSteps - 1 || ks == ksteps - 1) {
          const int mt = static_cast<int>(mins % kMins);
          const int b = static_cast<int>(turn % kBuffers<kRows>);
          ok = tc::MbarWait(&sh->tmem_empty[b], ((turn / kBuffers<kRows>) & 1u) ^ 1u);
          if constexpr (kSlab) ok = ok && tc::MbarWait(&sh->minw_full[mt], (mins / kMins) & 1);
          if (!__all_sync(0xffffffffu, ok)) {
            ok = false;
            break;
          }
          tc::TcFenceAfter();
          if (elected) {
            const std::uint64_t myd = tc::SmemDesc(min_y + (mt * kMinTileBytes), true, 1024);
            const std::uint64_t mwd = tc::SmemDesc(min_w + (mt * kMinTileBytes), true, 1024);
            const int last = (ks % kMinSteps) / 4;
            for (int q = 0; q <= last; ++q) {  // 32 bytes along the swizzled row each
              tc::MmaF16(tmem + (b * kBufferColumns<kRows>), myd + (q * 2), mwd + (q * 2), fdesc, q > 0);
            }
            tc::TcCommit(&sh->tmem_full[b]);
            tc::TcCommit(&sh->min_free[mt]);
          }
          ++turn;
          ++mins;
        }
        __syncwarp();
      }
    }
    if (!ok && elected) give_up();
  } else {
    // ------------------------------------------------------------ epilogue
    // acc += C * (d8 * d sc) for 64 rows a thread, 16 at a time: a piece is two TMEM loads, the
    // integers and the scale products the tensor core formed beside them, one conversion a value
    // and one packed multiply-add a pair.
    const int ew = warp - kFirstEpilogueWarp;
    const int quadrant = warp & 3;          // TMEM lanes this warp may touch
    const int rowgroup = ew >> 2;           // which kEpilogueRows weight rows
    const int tt = (quadrant * 32) + lane;  // token of the tile
    const std::uint32_t base =
        tmem + (static_cast<std::uint32_t>(quadrant * 32) << 16) + (rowgroup * kEpilogueRows<kRows>);
    std::uint64_t acc2[kEpilogueRows<kRows> / 2];  // rows 2i, 2i + 1
    std::uint32_t ca[16], sa[16], cb[16], sb[16];  // two pieces
    std::uint32_t turn = 0;
    bool ok = true, ahead = false;  // ahead: the group's first piece is already on its way
    const auto fold = [&](int piece, const std::uint32_t (&c)[16], const std::uint32_t (&s)[16]) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        acc2[(piece * 8) + i] =
            Fma2(Pack2(__int2float_rn(static_cast<int>(c[2 * i])), __int2float_rn(static_cast<int>(c[(2 * i) + 1]))),
                 Pack2(__uint_as_float(s[2 * i]), __uint_as_float(s[(2 * i) + 1])),
                 acc2[(piece * 8) + i]);
      }
    };
    const auto check = [&](int group, int piece, int col, int row0, const std::uint32_t (&c)[16]) {
      // verification: the exact group sums, before any float touches them
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const int row = row0 + (rowgroup * kEpilogueRows<kRows>) + (piece * 16) + j;
        if (row < a.nrows) {
          p.sums[((static_cast<std::size_t>(col) * a.nrows + row) * (a.k / 32)) + group] =
              static_cast<std::int32_t>(c[j]);
        }
      }
    };
    const auto load = [&](std::uint32_t from, std::uint32_t (&c)[16], std::uint32_t (&s)[16]) {
      tc::TmemLoad16(from, c);
      tc::TmemLoad16(from + kRows, s);
    };
    const int groups = ksteps * 4;
    for (std::int64_t i = blockIdx.x; i < tiles && ok && !*abort_flag; i += gridDim.x) {
      const Tile tile = tile_at(i);
      const int c_end = tile.c_end;
      if (tile.col0 >= c_end) continue;
      const int row0 = tile.row_tile * kRows;
      const int col = tile.col0 + tt;  // this thread's sorted column
#pragma unroll
      for (int j = 0; j < kEpilogueRows<kRows> / 2; ++j) acc2[j] = 0ull;
      // A k-step's four groups a turn of the loop: 4096 tokens x 4096 -> 14336 1320 us with one, 1233
      // with two, 1211 with four, 1347 with eight, whose code misses the instruction cache.  (The min
      // terms take a buffer's turn too, so buffers and parities stay run-time values.)
#pragma unroll 4
      for (int g = 0; g < groups; ++g) {
        const int b = static_cast<int>(turn % kBuffers<kRows>);
        const std::uint32_t at = base + (b * kBufferColumns<kRows>);
        if (!ahead) {
          ok = tc::MbarWait(&sh->tmem_full[b], (turn / kBuffers<kRows>) & 1u);
          if (!__all_sync(0xffffffffu, ok)) {
            ok = false;
            break;
          }
          tc::TcFenceAfter();
          load(at, ca, sa);
        }
        ++turn;
        constexpr int kPieces = kEpilogueRows<kRows> / 16;
#pragma unroll
        for (int piece = 0; piece < kPieces; piece += 2) {
          PieceWait(ca, sa);
          load(at + (16 * piece) + 16, cb, sb);
          if constexpr (kSums) {
            if (col < c_end) check(g, piece, col, row0, ca);
          }
          fold(piece, ca, sa);
          PieceWait(cb, sb);
          if (piece + 2 == kPieces) break;
          load(at + (16 * piece) + 32, ca, sa);
          if constexpr (kSums) {
            if (col < c_end) check(g, piece + 1, col, row0, cb);
          }
          fold(piece + 1, cb, sb);
        }
        // The buffer goes back to the tensor core; the next group's first piece, if it is there
        // already, is requested under this one's last fold.
        tc::TcFenceBefore();
        __syncwarp();
        if (lane == 0) tc::MbarArrive(&sh->tmem_empty[b]);
        const bool tail = (g & 63) == 63 || g == groups - 1;
        ahead = false;
        if (!tail) {
          const int nb = static_cast<int>(turn % kBuffers<kRows>);
          ahead = __all_sync(0xffffffffu, tc::MbarTest(&sh->tmem_full[nb], (turn / kBuffers<kRows>) & 1u));
          if (ahead) {
            tc::TcFenceAfter();
            load(base + (nb * kBufferColumns<kRows>), ca, sa);
          }
        }
        if constexpr (kSums) {
          if (col < c_end) check(g, kPieces - 1, col, row0, cb);
        }
        fold(kPieces - 1, cb, sb);
        if (tail) {
          // The min terms of 64 groups: sum of (-dmin * m) * s8, taken by the tensor core.
          const int mb = static_cast<int>(turn % kBuffers<kRows>);
          ok = tc::MbarWait(&sh->tmem_full[mb], (turn / kBuffers<kRows>) & 1u);
          if (!__all_sync(0xffffffffu, ok)) {
            ok = false;
            break;
          }
          tc::TcFenceAfter();
          ++turn;
#pragma unroll
          for (int piece = 0; piece < kPieces; ++piece) {
            tc::TmemLoad16(base + (mb * kBufferColumns<kRows>) + (piece * 16), ca);
            tc::TmemLoadWait16(ca);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              acc2[(piece * 8) + i] =
                  Add2(Pack2(__uint_as_float(ca[2 * i]), __uint_as_float(ca[(2 * i) + 1])), acc2[(piece * 8) + i]);
            }
          }
          tc::TcFenceBefore();
          __syncwarp();
          if (lane == 0) tc::MbarArrive(&sh->tmem_empty[mb]);
        }
      }
      if (!ok && lane == 0) give_up();
      float acc[kEpilogueRows<kRows>];
#pragma unroll
      for (int i = 0; i < kEpilogueRows<kRows> / 2; ++i) Unpack2(acc2[i], acc[2 * i], acc[(2 * i) + 1]);
      const int first = row0 + (rowgroup * kEpilogueRows<kRows>);
      const bool glu = kRows == kTileRows && p.glu_out != nullptr;
      if constexpr (kRows == kTileRows) {
        // The thread's 64 rows are twice 16 gate rows then the 16 up rows of the same outputs: one
        // Q8_1-MMQ group of 32 outputs, whose scale and sum are formed exactly as the quantizer
        // kernel does (eight lanes of four values, xor tree 4, 2, 1).
        if (glu && ok && col < c_end && first < a.nrows) {
          float h[32], part[8], amax = 0.0f;
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            const int gate = ((j >> 4) * 32) + (j & 15);
            h[j] = Glu(p.glu, acc[gate], acc[gate + 16], p.limit);
            amax = fmaxf(amax, fabsf(h[j]));
          }
#pragma unroll
          for (int l = 0; l < 8; ++l) {
            part[l] = ((h[4 * l] + h[(4 * l) + 1]) + h[(4 * l) + 2]) + h[(4 * l) + 3];
          }
          const float sum = ((part[0] + part[4]) + (part[2] + part[6])) +
                            ((part[1] + part[5]) + (part[3] + part[7]));
          std::uint32_t packed[8] = {0, 0, 0, 0, 0, 0, 0, 0};
          float d = 0.0f;
          if (amax > 0.0f) {
            const float d_inv = 127.0f / amax;
#pragma unroll
            for (int j = 0; j < 32; ++j) {
              const int q = static_cast<int>(roundf(h[j] * d_inv));
              packed[j >> 2] |= (static_cast<std::uint32_t>(q) & 0xffu) << (8 * (j & 3));
            }
            d = 1.0f / d_inv;
          }
          const int out_first = first / 2;  // this thread's first GLU output
          std::uint8_t* block = p.glu_out + (((static_cast<std::size_t>(out_first >> 7) * a.ncols) + col) * 144);
          const int at = out_first & 127;
          auto* codes = reinterpret_cast<uint4*>(block + 16 + at);
          codes[0] = make_uint4(packed[0], packed[1], packed[2], packed[3]);
          codes[1] = make_uint4(packed[4], packed[5], packed[6], packed[7]);
          *reinterpret_cast<std::uint32_t*>(block + ((at >> 5) * 4)) =
              static_cast<std::uint32_t>(__half_as_ushort(__float2half_rn(d))) |
              (static_cast<std::uint32_t>(__half_as_ushort(__float2half_rn(sum))) << 16);
        }
      }
      if (!glu && ok && col < c_end) {
        const int dst_col = a.ids_dst != nullptr ? a.ids_dst[col] : col;
        float* out = a.dst + (static_cast<std::size_t>(dst_col) * a.dst_col_stride) + first;
        // 256 contiguous bytes a thread: 128-bit stores when the output allows them
        const bool vector = (a.dst_col_stride % 4 == 0) &&
                            (reinterpret_cast<std::uintptr_t>(a.dst) % 16 == 0);
#pragma unroll  // fully: a dynamic index would put acc[] in local memory
        for (int v = 0; v < kEpilogueRows<kRows> / 4; ++v) {
          if (vector && first + (4 * v) + 4 <= a.nrows) {
            reinterpret_cast<float4*>(out)[v] =
                make_float4(acc[4 * v], acc[(4 * v) + 1], acc[(4 * v) + 2], acc[(4 * v) + 3]);
          } else {
#pragma unroll
            for (int j = 4 * v; j < (4 * v) + 4; ++j) {
              if (first + j < a.nrows) out[j] = acc[j];
            }
          }
        }
      }
    }
  }

  tc::TcFenceBefore();
  __syncthreads();
  if (warp == kMmaWarp) {
    tc::TcFenceAfter();
    tc::TmemDealloc(tmem, 512);
  }
}

int CheckDesc(const Desc& d, bool no_f32_output) {
  if (d.type != LLMP_B200_TYPE_Q4_K) {
    return Reject("mmq: weight type %d is not one this build computes (Q4_K)", d.type);
  }
  if ((d.w == nullptr && d.w_slab == nullptr) || d.y == nullptr ||
      (d.dst == nullptr && !no_f32_output) || d.k < 256 ||
      d.k % 256 != 0 || d.nrows < 1 || d.ncols < 1) {
    return Reject("mmq: Q4_K weights [k, n] (blocks or slab), Q8_1-MMQ activations of ncols columns, "
                  "an F32 output; k a positive multiple of 256");
  }
  if (d.stride_row < d.k / 256 || d.stride_expert < 0 ||
      (d.dst_col_stride < d.nrows && !no_f32_output)) {
    return Reject("mmq: strides must cover a row");
  }
  if ((d.w != nullptr && !Aligned(d.w, 16)) || !Aligned(d.y, 16) || !Aligned(d.dst, 4) ||
      (d.w_slab != nullptr && !Aligned(d.w_slab, 256)) ||
      (d.scratch != nullptr && !Aligned(d.scratch, 256))) {
    return Reject("mmq: weights and activation blocks 16-byte aligned; slab and scratch 256");
  }
  if (d.expert_bounds == nullptr && d.experts > 1) {
    return Reject("mmq: expert bounds exactly with experts");
  }
  if (d.expert_bounds != nullptr && (d.experts < 1 || d.experts > 65535)) {
    return Reject("mmq: 1 to 65535 experts");
  }
  return 0;
}

template <typename Fn>
bool Encode3D(CUtensorMap* map, Fn encode, const void* base, cuuint64_t d0, cuuint64_t d1,
              cuuint64_t d2, cuuint64_t s1, cuuint64_t s2, cuuint32_t b0, cuuint32_t b1,
              cuuint32_t b2, bool swizzle, CUtensorMapL2promotion promotion) {
  const cuuint64_t dims[3] = {d0, d1, d2};
  const cuuint64_t strides[2] = {s1, s2};
  const cuuint32_t box[3] = {b0, b1, b2};
  const cuuint32_t elem[3] = {1, 1, 1};
  return encode(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void*>(base), dims, strides, box,
                elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                swizzle ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE, promotion,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

int Relayout(const void* w, int n, int k, std::int64_t stride_row, std::int64_t stride_expert,
             int experts, void* slab, void* stream, int glu_inter = 0) {
  const Slab layout = SlabOf(n, k, experts);
  const std::int64_t items = static_cast<std::int64_t>(experts) * layout.row_tiles * 4 * (k / 256);
  const std::int64_t grid = (items + 7) / 8;
  if (grid > 0x7fffffffLL) return Reject("q4k_relayout: more blocks than a grid holds");
  const cudaError_t e = LaunchPdl(RelayoutQ4KKernel, dim3(static_cast<unsigned>(grid)), dim3(256), 0,
                                  static_cast<cudaStream_t>(stream),
                                  static_cast<const std::uint8_t*>(w), n, k, stride_row, stride_expert,
                                  experts, static_cast<std::uint8_t*>(slab), layout, glu_inter);
  if (e != cudaSuccess) return Failed(e, "q4k_relayout launch");
  return 0;
}

}  // namespace

int LaunchMmq(const llmp_b200_mmq_desc& d, const std::int32_t* worklist, int max_tiles,
              void* stream, std::int32_t* sums, const MmqGlu* glu) {
  if (const int status = CheckDesc(d, glu != nullptr); status != 0) return status;
  if (glu != nullptr) {
    if (d.w_slab == nullptr || glu->blocks == nullptr || d.nrows % 64 != 0 || d.ids_dst != nullptr ||
        sums != nullptr || !Aligned(glu->blocks, 16) || glu->glu < LLMP_B200_GLU_SWIGLU ||
        glu->glu > LLMP_B200_GLU_GEGLU || (glu->glu == LLMP_B200_GLU_GEGLU && glu->limit != 0.0f)) {
      return Reject("mmq_glu: a slab of interleaved gate / up rows (llmp_b200_q4k_relayout_glu), rows a "
                    "multiple of 64, no output scatter, 16-byte aligned output blocks, a GLU");
    }
  }
  if (const int status = DeviceStatus(); status != 0) return status;
  const tc::EncodeTiledFn encode = tc::EncodeTiled();
  if (encode == nullptr) return Reject("mmq: the driver has no tensor-map encoder");
  const int experts = d.expert_bounds != nullptr ? d.experts : 1;
  // The weights' slab: the caller's (relayout at load time), or built now in the
  // caller's scratch; without either the kernel decodes the raw blocks itself.
  const std::uint8_t* slab = static_cast<const std::uint8_t*>(d.w_slab);
  bool queued = false;
  if (slab == nullptr && d.scratch != nullptr) {
    const int status = Relayout(d.w, d.nrows, d.k, d.stride_row,
                                experts > 1 ? d.stride_expert
                                            : static_cast<std::int64_t>(d.stride_row) * d.nrows,
                                experts, d.scratch, stream);
    if (status != 0) return status;
    slab = static_cast<const std::uint8_t*>(d.scratch);
    queued = true;
  }
  const auto fail = [&](int status) { return (queued && status > 0) ? -status : status; };
  const Slab layout = SlabOf(d.nrows, d.k, experts);
  // Tiles of 64 weight rows for a dense product whose tiles of 64 all run at once: a tile is 0.7 to 0.8 of
  // the time of one of 128, so they pay where twice as many are still one wave (from blocks and from a slab,
  // 60 tokens x 4096 -> 2048 56.5 -> 40.0 and 49.5 -> 37.4 us, 200 x 2560 -> 4096 40.7 -> 30.9 and 38.0 -> 29.8;
  // three waves against two, 203 x 2560 -> 10240: 80.7 / 78.3 and 75.5 / 70.3).
  const std::int64_t half_tiles = static_cast<std::int64_t>((d.nrows + 63) / 64) * ((d.ncols + kTileCols - 1) / kTileCols);
  const bool narrow = worklist == nullptr && d.expert_bounds == nullptr && sums == nullptr && glu == nullptr &&
                      half_tiles <= SmCount();
  const cuuint32_t box_rows = narrow ? 64 : kTileRows;
  CUtensorMap map_y, map_w, map_h, map_mw;
  if (!Encode3D(&map_y, encode, static_cast<const std::uint8_t*>(d.y) + 16, 128,
                static_cast<cuuint64_t>(d.ncols), static_cast<cuuint64_t>(d.k / 128), 144,
                static_cast<cuuint64_t>(d.ncols) * 144, 128, kTileCols, 1, true,
                CU_TENSOR_MAP_L2_PROMOTION_L2_256B)) {
    return fail(Reject("mmq: the driver refused a tensor map for the activation blocks"));
  }
  // The activation blocks' 16-byte headers [k / 128][col]: a box is 128 tokens, two k-steps.
  if (!Encode3D(&map_h, encode, d.y, 16, static_cast<cuuint64_t>(d.ncols),
                static_cast<cuuint64_t>(d.k / 128), 144, static_cast<cuuint64_t>(d.ncols) * 144, 16,
                kTileCols, 2, false, CU_TENSOR_MAP_L2_PROMOTION_NONE)) {
    return fail(Reject("mmq: the driver refused a tensor map for the activation headers"));
  }
  if (slab != nullptr) {
    // int8 codes [expert][row][k]: a box is 128 rows of one k-step, swizzled for the MMA.
    if (!Encode3D(&map_w, encode, slab + layout.codes, static_cast<cuuint64_t>(d.k),
                  static_cast<cuuint64_t>(d.nrows), static_cast<cuuint64_t>(experts),
                  static_cast<cuuint64_t>(d.k), static_cast<cuuint64_t>(d.k) * d.nrows, kBK,
                  box_rows, 1, true, CU_TENSOR_MAP_L2_PROMOTION_L2_256B) ||
        !Encode3D(&map_mw, encode, slab + layout.mw, static_cast<cuuint64_t>(layout.gpad) * 2,
                  static_cast<cuuint64_t>(d.nrows), static_cast<cuuint64_t>(experts),
                  static_cast<cuuint64_t>(layout.gpad) * 2,
                  static_cast<cuuint64_t>(layout.gpad) * 2 * d.nrows, 128, box_rows, 1, true,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B)) {
      return fail(Reject("mmq: the driver refused a tensor map for the weight slab"));
    }
  } else {
    // The weights as bytes [expert][row][k / 256 * 144]: a box is one block of 128 rows.
    const cuuint64_t row_pitch = static_cast<cuuint64_t>(d.stride_row) * 144;
    const cuuint64_t expert_pitch = experts > 1 ? static_cast<cuuint64_t>(d.stride_expert) * 144
                                                : row_pitch * static_cast<cuuint64_t>(d.nrows);
    if (!Encode3D(&map_w, encode, d.w, static_cast<cuuint64_t>(d.k / 256) * 144,
                  static_cast<cuuint64_t>(d.nrows), static_cast<cuuint64_t>(experts), row_pitch,
                  expert_pitch, 144, box_rows, 1, false, CU_TENSOR_MAP_L2_PROMOTION_L2_256B)) {
      return fail(Reject("mmq: the driver refused a tensor map for the weight blocks"));
    }
    map_mw = map_w;  // unused
  }
  Params p{};
  p.a = d;
  p.worklist = worklist;
  p.faults = FaultCounter();
  if (p.faults == nullptr) return fail(Reject("mmq: no fault counter on this device"));
  p.ax = slab != nullptr ? reinterpret_cast<const float*>(slab + layout.ax) : nullptr;
  p.ax_ksteps = layout.ksteps;
  p.ax_row_tiles = layout.row_tiles;
  p.sums = sums;
  if (glu != nullptr) {
    p.glu_out = static_cast<std::uint8_t*>(glu->blocks);
    p.glu = glu->glu;
    p.limit = glu->limit;
  }
  static thread_local int configured_device = -1;
  int device = -1;
  cudaGetDevice(&device);
  if (configured_device != device) {
    const auto allow = [](const void* kernel, int bytes) {
      return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    };
    cudaError_t e = allow(reinterpret_cast<const void*>(&MmqQ4KKernel<false, false, kTileRows>), kSmem<false>);
    if (e == cudaSuccess) e = allow(reinterpret_cast<const void*>(&MmqQ4KKernel<true, false, kTileRows>), kSmem<true>);
    if (e == cudaSuccess) e = allow(reinterpret_cast<const void*>(&MmqQ4KKernel<false, true, kTileRows>), kSmem<false>);
    if (e == cudaSuccess) e = allow(reinterpret_cast<const void*>(&MmqQ4KKernel<true, true, kTileRows>), kSmem<true>);
    if (e == cudaSuccess) e = allow(reinterpret_cast<const void*>(&MmqQ4KKernel<false, false, 64>), kSmem<false>);
    if (e == cudaSuccess) e = allow(reinterpret_cast<const void*>(&MmqQ4KKernel<true, false, 64>), kSmem<true>);
    if (e != cudaSuccess) return fail(Failed(e, "mmq attribute"));
    configured_device = device;
  }
  std::int64_t tiles = (d.nrows + static_cast<int>(box_rows) - 1) / static_cast<int>(box_rows);
  if (worklist != nullptr) {
    if (max_tiles < 1) return fail(Reject("mmq: a worklist needs its capacity"));
    p.col_tiles = max_tiles;
  } else {
    const int max_cols = d.expert_bounds != nullptr ? d.max_cols_per_expert : d.ncols;
    if (max_cols < 1) return fail(Reject("mmq: max_cols_per_expert >= 1 with experts"));
    p.col_tiles = (max_cols + kTileCols - 1) / kTileCols;
    tiles *= experts;
  }
  if (p.col_tiles > 65535) return fail(Reject("mmq: more column tiles than a grid holds"));
  tiles *= p.col_tiles;
  // A CTA an SM (its shared memory and all of the SM's tensor memory), persistent: the next tile's
  // operands and first groups come in under a tile's write-back.
  const dim3 grid(static_cast<unsigned>(std::min<std::int64_t>(tiles, SmCount())));
  auto* s = static_cast<cudaStream_t>(stream);
  const auto kernel = narrow ? (slab != nullptr ? &MmqQ4KKernel<true, false, 64> : &MmqQ4KKernel<false, false, 64>)
                      : slab != nullptr ? (sums != nullptr ? &MmqQ4KKernel<true, true, kTileRows> : &MmqQ4KKernel<true, false, kTileRows>)
                                      : (sums != nullptr ? &MmqQ4KKernel<false, true, kTileRows> : &MmqQ4KKernel<false, false, kTileRows>);
  const cudaError_t e = LaunchPdl(kernel, grid, dim3(kThreads), slab != nullptr ? kSmem<true> : kSmem<false>, s,
                                  map_y, map_w, map_h, map_mw, p);
  if (e != cudaSuccess) return Failed(e, "mmq launch");
  return 0;
}

}  // namespace llmp_b200

extern "C" {

int64_t llmp_b200_mmq_q8_1_bytes(int64_t k, int64_t cols) { return (k / 128) * cols * 144; }

int llmp_b200_mmq_quantize(const void* x, int is_bf16, int64_t row_stride, int64_t k, int64_t cols,
                           const int32_t* ids_src, void* out, void* stream) {
  using namespace llmp_b200;
  if (x == nullptr || out == nullptr || k < 128 || k % 128 != 0 || cols < 1 || row_stride < k) {
    return Reject("mmq.quantize: [k, rows] input with k a positive multiple of 128, cols >= 1");
  }
  const int elem = is_bf16 ? 2 : 4;
  if (!Aligned(x, 16) || (row_stride * elem) % 16 != 0 || !Aligned(out, 16)) {
    return Reject("mmq.quantize: input rows and output 16-byte aligned");
  }
  if (const int status = DeviceStatus(); status != 0) return status;
  return is_bf16 ? QuantizeMmq<true, false>(x, row_stride, k, cols, ids_src, nullptr, 0, out, stream)
                 : QuantizeMmq<false, false>(x, row_stride, k, cols, ids_src, nullptr, 0, out, stream);
}

int llmp_b200_mmq_quantize_slots(const void* x, int is_bf16, int64_t row_stride, int64_t k, int64_t tokens,
                                 const int32_t* position, int used, void* out, void* stream) {
  using namespace llmp_b200;
  if (x == nullptr || position == nullptr || out == nullptr || k < 128 || k % 128 != 0 || tokens < 1 ||
      used < 1 || row_stride < k) {
    return Reject("mmq.quantize_slots: [k, tokens] input with k a positive multiple of 128, [tokens, used] "
                  "positions");
  }
  const int elem = is_bf16 ? 2 : 4;
  if (!Aligned(x, 16) || (row_stride * elem) % 16 != 0 || !Aligned(out, 16) || !Aligned(position, 4)) {
    return Reject("mmq.quantize_slots: input rows and output 16-byte aligned, positions 4");
  }
  if (const int status = DeviceStatus(); status != 0) return status;
  return is_bf16 ? QuantizeMmq<true, true>(x, row_stride, k, tokens, nullptr, position, used, out, stream)
                 : QuantizeMmq<false, true>(x, row_stride, k, tokens, nullptr, position, used, out, stream);
}

size_t llmp_b200_q4k_slab_bytes(int nrows, int k, int experts) {
  if (nrows < 1 || k < 256 || k % 256 != 0 || experts < 1) return 0;
  return llmp_b200::SlabOf(nrows, k, experts).total;
}

int llmp_b200_q4k_relayout(const void* w, int nrows, int k, int stride_row, int64_t stride_expert,
                           int experts, void* slab, void* stream) {
  using namespace llmp_b200;
  if (w == nullptr || slab == nullptr || nrows < 1 || k < 256 || k % 256 != 0 || experts < 1 ||
      stride_row < k / 256 || (experts > 1 && stride_expert < static_cast<int64_t>(stride_row) * nrows)) {
    return Reject("q4k_relayout: Q4_K blocks [experts][n][k / 256], k a positive multiple of 256, "
                  "strides that cover a row and an expert, and a slab");
  }
  if (!Aligned(w, 16) || !Aligned(slab, 256)) {
    return Reject("q4k_relayout: blocks 16-byte aligned, the slab 256");
  }
  if (const int status = DeviceStatus(); status != 0) return status;
  return Relayout(w, nrows, k, stride_row, stride_expert, experts, slab, stream);
}

size_t llmp_b200_mmq_scratch(const llmp_b200_mmq_desc* desc, int sms) {
  (void)sms;
  if (desc == nullptr || desc->w_slab != nullptr) return 0;
  const int experts = desc->expert_bounds != nullptr ? desc->experts : 1;
  return llmp_b200_q4k_slab_bytes(desc->nrows, desc->k, experts);
}

int llmp_b200_mmq(const llmp_b200_mmq_desc* desc, int sms, void* stream) {
  (void)sms;
  if (desc == nullptr) return llmp_b200::Reject("mmq: null descriptor");
  return llmp_b200::LaunchMmq(*desc, nullptr, 0, stream, nullptr);
}

int llmp_b200_q4k_relayout_glu(const void* w, int inter, int k, int stride_row, int64_t stride_expert,
                               int experts, void* slab, void* stream) {
  using namespace llmp_b200;
  if (w == nullptr || slab == nullptr || inter < 32 || inter % 32 != 0 || k < 256 || k % 256 != 0 ||
      experts < 1 || stride_row < k / 256 ||
      (experts > 1 && stride_expert < static_cast<int64_t>(stride_row) * 2 * inter)) {
    return Reject("q4k_relayout_glu: Q4_K blocks [experts][2 * inter][k / 256] (gate rows, then up "
                  "rows), inter a positive multiple of 32, k of 256, and a slab");
  }
  if (!Aligned(w, 16) || !Aligned(slab, 256)) {
    return Reject("q4k_relayout_glu: blocks 16-byte aligned, the slab 256");
  }
  if (const int status = DeviceStatus(); status != 0) return status;
  return Relayout(w, 2 * inter, k, stride_row, stride_expert, experts, slab, stream, inter);
}

int llmp_b200_mmq_glu(const llmp_b200_mmq_desc* desc, int glu, float limit, void* blocks,
                      void* stream) {
  using namespace llmp_b200;
  if (desc == nullptr) return Reject("mmq_glu: null descriptor");
  const MmqGlu g{blocks, glu, limit};
  return LaunchMmq(*desc, nullptr, 0, stream, nullptr, &g);
}

int llmp_b200_mmq_block_sums(const llmp_b200_mmq_desc* desc, int32_t* sums, void* stream) {
  using namespace llmp_b200;
  if (desc == nullptr || sums == nullptr) return Reject("mmq_block_sums: a descriptor and an output");
  if (desc->expert_bounds != nullptr || desc->ids_dst != nullptr) {
    return Reject("mmq_block_sums: the dense product only");
  }
  return LaunchMmq(*desc, nullptr, 0, stream, sums);
}

}  // extern "C"
