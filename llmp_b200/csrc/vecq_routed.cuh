// Routed Q4_K llmp.vecq for a batch of tokens (72 pairs and more): every expert that a token names is
// streamed once for up to eight of the (token, slot) pairs that name it, the int8 products on
// the tensor cores (mma.sync m16n8k32, u8 x s8 -> s32) with the MMA's eight columns the pairs.
// Interface and sums' contract are the reference's (src/kernels/ggml/vecq.h:23-49,
// vecq.cu:457-665); the ownership of an expert (vecq.cu:514-546) is by a list here.
//
// What bounds it: a tile's latency.  A block of 128 experts, top 8, 2048 x 768 at 64 tokens takes
// 147 us; its products' weights are 52 us of the measured copy rate and their instructions 64 us of
// issue slots (443 and 554 warp instructions a 16-row x 256-value unit of gate | up and down, the
// lists, the staging and the meetings counted), and of a warp's time between two instructions 41
// and 30 % goes to the group's barrier.  The register-staged kernel (vecq_impl.cuh) launches a
// grid row for every (token, slot) pair, most of which leave after scanning the ids, and its dot
// products take an instruction for four values of ONE pair.
//
//   * One persistent CTA an SM.  It builds the list of distinct experts and their pairs in shared
//     memory (a hash table for the counts, a warp's scan over the pairs in order for the list; every
//     CTA holds the same list, in the same order), and takes an equal, contiguous share of the units (expert,
//     pass of eight pairs, 16-row tile): at most a few changes of expert a CTA.
//   * Warps form groups; a group multiplies one tile at a time, its warps splitting the row's
//     super-block columns, and owns a ring of tiles brought by bulk copies (the group's barrier
//     after a tile is also what frees its stage: no second set of mbarriers).
//   * The fragments are those of the dense token-column kernel (vecq_rowmma.cuh); chunk by chunk
//     for both matrices, so a chunk's activations and scales are read once for gate and up.  The
//     odd sub-blocks' codes stay in place as 16 x code and 1/16 goes to the token's scale: both
//     exact.
//   * A pair's result does not depend on its company or on its place among the pairs.
//   * Every mbarrier wait is bounded and reports through the fault counter; nothing of a tile
//     that did not land is stored, and the group that waited for it requests no more and waits
//     (bounded again) for what it has in flight before the CTA may end.
#ifndef LLMP_B200_CSRC_VECQ_ROUTED_CUH_
#define LLMP_B200_CSRC_VECQ_ROUTED_CUH_

#include "vecq_unit.cuh"

namespace llmp_b200 {
namespace vecq {

constexpr int kRoutedFewest = 72;       // pairs from which a batch takes this kernel
constexpr int kRoutedWarps = 16;        // 128 registers a thread
constexpr int kRoutedPairs = kUnitTokens;  // pairs a pass
constexpr int kRoutedTile = 16;         // rows a tile
constexpr int kRoutedPartialRows = 18;  // a pair's pitch in the partial sums: no two lanes of a
                                        // half-warp's 64-bit stores on one bank
constexpr int kRoutedMaxStages = 64;    // of all groups
constexpr int kRoutedHash = 2048;       // entries, for at most kMaxPairs experts

struct RoutedPlan {
  int grid;
  int groups;      // groups of warps
  int col_groups;  // warps a group: they split a row's super-block columns
  int stages;      // tiles a group's ring holds
  int columns;     // k / 256
  int tiles;       // 16-row tiles of an expert
  int pitch;       // bytes between staged rows
  int packed;      // one bulk copy a tile and matrix (pitch == a row's bytes)
  int acts_bytes;  // the pass's staged activations
  int smem_bytes;
  unsigned int* faults;
};

// The list of the pairs by expert; in shared memory, after the staged operands.
struct RoutedList {
  int expert[kMaxPairs];           // distinct experts, in the order of their first pairs
  int pass_end[kMaxPairs];         // passes of experts 0 .. i
  std::uint16_t start[kMaxPairs];  // an expert's first pair in `pairs`
  std::uint16_t count[kMaxPairs];
  std::uint16_t pairs[kMaxPairs];  // token << 8 | slot
  int experts, passes;
};
// What building it needs; lies over the ring before the first copy is requested.
struct RoutedHash {
  int key[kRoutedHash];
  int first[kRoutedHash];
  int count[kRoutedHash];
  int cursor[kRoutedHash];
  std::uint16_t start[kRoutedHash];
  std::uint16_t slot[kMaxPairs];
  std::uint16_t loose[kMaxPairs];
};
constexpr int kRoutedEmpty = static_cast<int>(0x80000000u);  // no expert's index

template <bool kGlu>
__global__ void __launch_bounds__(kRoutedWarps * 32, 1)
VecQRoutedKernel(const Desc a, const RoutedPlan plan) {
  constexpr int kMats = kGlu ? 2 : 1;
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ __align__(8) std::uint64_t full[kRoutedMaxStages];
  __shared__ int abort_flag;

  const int tid = static_cast<int>(threadIdx.x);
  const int threads = static_cast<int>(blockDim.x);
  const int warp = tid >> 5;
  const int lane = tid & 31;
  const int g = lane >> 2;  // rows g and g + 8; column g of B
  const int t = lane & 3;
  const int UR = plan.columns;
  const int wc = warp % plan.col_groups;
  const int group = warp / plan.col_groups;
  const int group_threads = plan.col_groups * 32;
  const int stage_bytes = kMats * kRoutedTile * plan.pitch;
  const int partial_floats = plan.col_groups * kRoutedPairs * kRoutedPartialRows * kMats;
  const std::uint32_t row_bytes = static_cast<std::uint32_t>(UR) * 144u;

  // smem: [the pass's activations][the groups' rings][the groups' partial sums, two each][list]
  unsigned char* acts = smem;
  const TokenActs layout(UR);
  unsigned char* rings = acts + plan.acts_bytes;
  unsigned char* ring = rings + (static_cast<std::size_t>(group) * plan.stages * stage_bytes);
  float* partials = reinterpret_cast<float*>(
      rings + (static_cast<std::size_t>(plan.groups) * plan.stages * stage_bytes));
  RoutedList* list = reinterpret_cast<RoutedList*>(partials + (plan.groups * 2 * partial_floats));
  float* partial = partials + (group * 2 * partial_floats);

  GridLaunchDependents();
  if (tid == 0) {
    for (int i = 0; i < plan.groups * plan.stages; ++i) MbarInit(&full[i], 1);
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  RoutedHash* hash = reinterpret_cast<RoutedHash*>(rings);
  for (int i = tid; i < kRoutedHash; i += threads) {
    hash->key[i] = kRoutedEmpty;
    hash->first[i] = kMaxPairs;
    hash->count[i] = 0;
    hash->cursor[i] = 0;
  }
  const int total = a.tokens * a.used;
  GridDependencyWait();  // the ids and the activations may be an earlier kernel's
  __syncthreads();
  for (int q = tid; q < total; q += threads) {
    const int id = a.ids[((q / a.used) * a.ids_stride) + (q % a.used)];
    std::uint32_t at = (static_cast<std::uint32_t>(id) * 2654435761u) >> 21;
    // at most kMaxPairs keys in twice as many entries: an empty one is found
    for (;;) {
      const int seen = atomicCAS(&hash->key[at], kRoutedEmpty, id);
      if (seen == kRoutedEmpty || seen == id) break;
      at = (at + 1) & (kRoutedHash - 1);
    }
    atomicMin(&hash->first[at], q);
    atomicAdd(&hash->count[at], 1);
    hash->slot[q] = static_cast<std::uint16_t>(at);
  }
  __syncthreads();
  if (warp == 0) {
    int experts = 0, before = 0;  // before: pairs (low half) and passes (high half) so far
    for (int q0 = 0; q0 < total; q0 += 32) {
      const int q = q0 + lane;
      const int at = q < total ? hash->slot[q] : 0;
      const bool owner = q < total && hash->first[at] == q;
      const int n = owner ? hash->count[at] : 0;
      const int mine = n | (((n + kRoutedPairs - 1) / kRoutedPairs) << 16);
      int sum = mine;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, sum, d);
        if (lane >= d) sum += up;
      }
      const unsigned owners = __ballot_sync(0xffffffffu, owner);
      if (owner) {
        const int i = experts + __popc(owners & ((1u << lane) - 1u));
        const int start = (before + sum - mine) & 0xffff;
        list->expert[i] = hash->key[at];
        list->pass_end[i] = (before + sum) >> 16;
        list->start[i] = static_cast<std::uint16_t>(start);
        list->count[i] = static_cast<std::uint16_t>(n);
        hash->start[at] = static_cast<std::uint16_t>(start);
      }
      experts += __popc(owners);
      before += __shfl_sync(0xffffffffu, sum, 31);
    }
    if (lane == 0) {
      list->experts = experts;
      list->passes = before >> 16;
    }
  }
  __syncthreads();
  // An expert's pairs in order (every CTA has to deal them to the same passes): dropped at the
  // expert's place as they come, then each counts those before it.
  for (int q = tid; q < total; q += threads) {
    const int at = hash->slot[q];
    hash->loose[hash->start[at] + atomicAdd(&hash->cursor[at], 1)] = static_cast<std::uint16_t>(q);
  }
  __syncthreads();
  for (int q = tid; q < total; q += threads) {
    const int at = hash->slot[q];
    const int start = hash->start[at], n = hash->count[at];
    int before = 0;
    for (int i = 0; i < n; ++i) before += hash->loose[start + i] < q ? 1 : 0;
    list->pairs[start + before] = static_cast<std::uint16_t>(((q / a.used) << 8) | (q % a.used));
  }
  FenceProxyAsync();  // the table's memory is the ring's from here on
  __syncthreads();

  const long units = static_cast<long>(list->passes) * plan.tiles;
  const long u0 = (units * blockIdx.x) / gridDim.x;
  const long u1 = (units * (blockIdx.x + 1)) / gridDim.x;
  // the expert whose passes hold pass `pass`
  const auto find = [&](int pass) {
    int lo = 0, hi = list->experts - 1;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (list->pass_end[mid] > pass) hi = mid; else lo = mid + 1;
    }
    return lo;
  };

  // Warp 0 of a group requests the group's tiles, in order: units u0 + group, + groups, ...
  long want = u0 + group;
  int want_pass = 0, want_tile = 0, want_expert = 0, want_stage = 0;
  if (wc == 0 && want < u1) {
    want_pass = static_cast<int>(want / plan.tiles);
    want_tile = static_cast<int>(want % plan.tiles);
    want_expert = find(want_pass);
  }
  long want_end = u1;  // nothing more is requested once a wait has run out
  const auto request = [&]() {
    if (want >= want_end) return;
    const int r0 = want_tile * kRoutedTile;
    const int n = min(kRoutedTile, a.nrows - r0);
    std::uint64_t* bar = &full[(group * plan.stages) + want_stage];
    unsigned char* to = ring + (static_cast<std::size_t>(want_stage) * stage_bytes);
    const std::size_t from =
        ((static_cast<std::size_t>(list->expert[want_expert]) * a.stride_expert) +
         (static_cast<std::size_t>(r0) * a.stride_row)) * 144;
    if (lane == 0) MbarExpectTx(bar, static_cast<std::uint32_t>(n) * row_bytes * kMats);
    __syncwarp();
    if (plan.packed) {
      if (lane < kMats) {
        BulkLoad(to + (static_cast<std::size_t>(lane) * kRoutedTile * plan.pitch),
                 static_cast<const std::uint8_t*>(lane == 0 ? a.w : a.g) + from,
                 static_cast<std::uint32_t>(n) * row_bytes, bar);
      }
    } else {
      const int m = lane / kRoutedTile, r = lane % kRoutedTile;
      if (m < kMats && r < n) {
        BulkLoad(to + ((static_cast<std::size_t>(m) * kRoutedTile + r) * plan.pitch),
                 static_cast<const std::uint8_t*>(m == 0 ? a.w : a.g) + from +
                     (static_cast<std::size_t>(r) * a.stride_row * 144),
                 row_bytes, bar);
      }
    }
    want += plan.groups;
    want_tile += plan.groups;
    while (want_tile >= plan.tiles && want < u1) {
      want_tile -= plan.tiles;
      ++want_pass;
      if (want_pass >= list->pass_end[want_expert]) ++want_expert;
    }
    if (++want_stage == plan.stages) want_stage = 0;
  };
  if (wc == 0) {
    for (int i = 0; i < plan.stages; ++i) request();
  }

  bool healthy = true;
  int turn = 0, stage = 0;
  std::uint32_t parity = 0;
  long unit = u0 + group;  // the group's next
  for (long u = u0; u < u1;) {
    // One expert's pass: its pairs' activations, then the CTA's tiles of it.
    const int pass = static_cast<int>(u / plan.tiles);
    const int e = find(pass);
    const int done = (pass - (e > 0 ? list->pass_end[e - 1] : 0)) * kRoutedPairs;
    const std::uint16_t* pairs = list->pairs + list->start[e] + done;
    const int live = min(kRoutedPairs, list->count[e] - done);
    const long first_unit = static_cast<long>(pass) * plan.tiles;
    const long end = min(u1, first_unit + plan.tiles);
    __syncthreads();  // the pass before has read its activations
    const int blocks = UR * 8;
    for (int i = tid; i < live * blocks; i += threads) {
      const int p = i / blocks, b = i - (p * blocks);
      const int pr = pairs[p];
      StageUnitBlock(acts, layout, p, b,
                     static_cast<const std::uint8_t*>(a.y) +
                         ((static_cast<std::size_t>(pr >> 8) * a.y_token +
                           static_cast<std::size_t>(pr & 0xff) * a.y_slot + b) * 36));
    }
    __syncthreads();

    const UnitLane at_lane(acts, layout, live, lane);
    for (; unit < end; unit += plan.groups, ++turn) {
      const int r0 = static_cast<int>(unit - first_unit) * kRoutedTile;
      const int rows = min(kRoutedTile, a.nrows - r0);
      if (healthy && lane == 0 && !MbarWait(&full[(group * plan.stages) + stage], parity)) {
        healthy = false;
        abort_flag = 1;
        atomicAdd(plan.faults, 1u);
      }
      healthy = __shfl_sync(0xffffffffu, healthy ? 1 : 0, 0) != 0;
      if (!healthy) want_end = 0;
      const unsigned char* rows_at = ring + (static_cast<std::size_t>(stage) * stage_bytes);
      // rows g and g + 8 of the tile, clamped into the matrix (the last tile may be short)
      const unsigned char* lo_at = rows_at + (min(g, rows - 1) * plan.pitch);
      const unsigned char* hi_at = rows_at + (min(g + 8, rows - 1) * plan.pitch);
      float sums[kMats][2][2];  // [matrix][row g / g + 8][pair 2t / 2t + 1]
#pragma unroll
      for (int m = 0; m < kMats; ++m)
#pragma unroll
        for (int h = 0; h < 2; ++h) sums[m][h][0] = sums[m][h][1] = 0.0f;
      for (int c = wc; healthy && c < UR; c += plan.col_groups) {
        const unsigned char *lo[kMats], *hi[kMats];
#pragma unroll
        for (int m = 0; m < kMats; ++m) {
          lo[m] = lo_at + (m * kRoutedTile * plan.pitch) + (c * 144);
          hi[m] = hi_at + (m * kRoutedTile * plan.pitch) + (c * 144);
        }
        TokenUnit<kMats>(lo, hi, at_lane, 8 * t, c, sums);
      }
      float* mine = partial + ((turn & 1) * partial_floats);
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          float* at = mine + ((((wc * kRoutedPairs) + (2 * t) + j) * kRoutedPartialRows + g + (8 * h)) * kMats);
          if constexpr (kGlu) {
            *reinterpret_cast<float2*>(at) = make_float2(sums[0][h][j], sums[1][h][j]);
          } else {
            *at = sums[0][h][j];
          }
        }
      // The group has read the stage and written its partial sums.  (The next tile's go to the
      // other half; that tile's barrier is behind every read of this half.)
      if (plan.col_groups == 1) {
        __syncwarp();
      } else {
        asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "r"(group_threads) : "memory");
      }
      if (wc == 0) {
        FenceProxyAsync();
        request();
      }
      const bool keep = *static_cast<volatile int*>(&abort_flag) == 0;
      for (int i = (wc * 32) + lane; i < kRoutedPairs * kRoutedTile; i += group_threads) {
        const int p = i / kRoutedTile, r = i % kRoutedTile;
        if (p >= live || r >= rows || !keep) continue;
        float v[kMats];
#pragma unroll
        for (int m = 0; m < kMats; ++m) {
          v[m] = SumColumns(mine + (((p * kRoutedPartialRows) + r) * kMats) + m, plan.col_groups,
                            kRoutedPairs * kRoutedPartialRows * kMats);
        }
        float* dst = a.dst + (static_cast<std::size_t>(pairs[p] >> 8) * a.dst_token) +
                     (static_cast<std::size_t>(pairs[p] & 0xff) * a.dst_slot) + r0 + r;
        if constexpr (kGlu) {
          *dst = Glu(a.glu, v[1], v[0], a.limit);
        } else {
          *dst = v[0];
        }
      }
      if (++stage == plan.stages) {
        stage = 0;
        parity ^= 1u;
      }
    }
    u = end;
  }
  if (wc == 0 && !healthy) {
    // what the group still has in flight must not outlive the CTA: its ring's last requests
    const long first = (static_cast<long>(list->passes) * plan.tiles * blockIdx.x) / gridDim.x + group;
    const long requested = (want - first) / plan.groups;
    for (long i = max(0L, requested - plan.stages); i < requested; ++i) {
      MbarWait(&full[(group * plan.stages) + static_cast<int>(i % plan.stages)],
               static_cast<std::uint32_t>(i / plan.stages) & 1u);
    }
  }
}

// Host: the geometry, or false if the product does not fit.
inline bool PlanRouted(const Desc& d, int sms, RoutedPlan* plan) {
  const int mats = d.glu != LLMP_B200_GLU_NONE ? 2 : 1;
  const int ur = d.ncols_x / 256;
  const int row_bytes = ur * 144;
  // Rows back to back when their pitch spreads four rows' 32 bytes over the banks with at most
  // two on one; else a copy a row, at a pitch of 32 bytes modulo 128.
  const bool packed = d.stride_row == ur && row_bytes % 64 != 0;
  plan->columns = ur;
  plan->tiles = (d.nrows + kRoutedTile - 1) / kRoutedTile;
  plan->packed = packed ? 1 : 0;
  plan->pitch = packed ? row_bytes : ((row_bytes + 127) / 128 * 128) + 32;
  plan->acts_bytes = TokenActs(ur).Bytes();
  const int stage = mats * kRoutedTile * plan->pitch;
  const int fixed = plan->acts_bytes + static_cast<int>(sizeof(RoutedList)) + 128;
  const int limit = 225 * 1024;
  double best = 0.0;
  for (int c = 1; c <= std::min(ur, kRoutedWarps); ++c) {
    const int groups = kRoutedWarps / c;
    if (c > 1 && groups > 15) continue;  // a named barrier a group
    const int partial = groups * 2 * c * kRoutedPairs * kRoutedPartialRows * mats * 4;
    const int room = limit - fixed - partial;
    if (room < 2 * groups * stage) continue;
    const int stages = std::min({room / (groups * stage), kRoutedMaxStages / groups, 8});
    if (groups * stages * stage < static_cast<int>(sizeof(RoutedHash))) continue;
    // tiles a unit of time: a column a warp, and about a third of one for the group's meeting
    const double score = groups / (((ur + c - 1) / c) + 0.3);
    if (score <= best * 1.02) continue;
    best = score;
    plan->groups = groups;
    plan->col_groups = c;
    plan->stages = stages;
    plan->smem_bytes = fixed + partial + (groups * stages * stage);
  }
  plan->grid = sms;
  plan->faults = FaultCounter();
  return best > 0.0 && plan->faults != nullptr;
}

cudaError_t LaunchRouted(const Desc& d, const RoutedPlan& plan, cudaStream_t stream);

}  // namespace vecq
}  // namespace llmp_b200

#endif  // LLMP_B200_CSRC_VECQ_ROUTED_CUH_
