// Measured ranks of the dense Q4_K llmp.vecq launch configurations on B200 (the role of the
// reference's src/kernels/ggml/measured_ranks.h and src/execution/rank_data.h: checked-in
// measurements that pick an implementation per shape; unmeasured shapes keep the ordinary
// rule).  Each row is the fastest configuration of one (k, n, fused GLU, tokens) product among
// the row-lane, row-MMA (sub-block columns and token columns), stream and generic kernels, each timed as a CUDA-graph replay over
// weight copies that together exceed the L2 (median of 6), on one B200 at 1,965 MHz; a
// configuration displaces the plain row-lane kernel only when it measured more than 3 %
// faster.  tests/test_vecq_gpu.py fails when a row names a configuration the library no
// longer has.
#ifndef LLMP_B200_CSRC_VECQ_RANKS_H_
#define LLMP_B200_CSRC_VECQ_RANKS_H_

namespace llmp_b200 {
namespace vecq {

struct MeasuredRank {
  int k, n, glu, tokens;  // tokens: the pass size 1, 2, 4 or 8 the row stands for
  const char* variant;
  float microseconds;
  int gbs;
};

constexpr MeasuredRank kMeasuredRanks[] = {
    // k, n, fused GLU, tokens, variant, microseconds a launch, GB/s of weight bytes
    {2560, 10240, 1, 1, "rowlane", 7.287f, 4047},
    {2560, 10240, 1, 2, "rowlane", 8.946f, 3297},
    {2560, 10240, 1, 4, "rowmma.t8", 11.400f, 2587},
    {2560, 10240, 1, 8, "rowmma.t8", 13.410f, 2199},
    {10240, 2560, 0, 1, "rowmma.c2", 5.213f, 2829},
    {10240, 2560, 0, 2, "rowlane", 7.483f, 1971},
    {10240, 2560, 0, 4, "rowmma.t8", 8.650f, 1705},
    {10240, 2560, 0, 8, "rowmma.t8", 10.730f, 1374},
    {4096, 4096, 0, 1, "rowlane", 4.016f, 2350},
    {4096, 4096, 0, 2, "rowmma.t8c2", 4.560f, 2070},
    {4096, 4096, 0, 4, "rowmma.t8c2", 5.020f, 1880},
    {4096, 4096, 0, 8, "rowmma.t8", 6.110f, 1545},
    {4096, 14336, 1, 1, "rowlane", 16.293f, 4055},
    {4096, 14336, 1, 2, "rowlane", 20.101f, 3286},
    {4096, 14336, 1, 4, "rowmma.t8", 24.420f, 2705},
    {4096, 14336, 1, 8, "rowmma.t8", 27.940f, 2364},
    {14336, 4096, 0, 1, "rowlane", 10.299f, 3207},
    {14336, 4096, 0, 2, "rowlane", 11.459f, 2882},
    {14336, 4096, 0, 4, "rowmma.t8", 13.860f, 2383},
    {14336, 4096, 0, 8, "rowlane", 26.141f, 1264},
    {2048, 2048, 0, 1, "rowlane", 2.075f, 1137},
    {2048, 2048, 0, 2, "rowlane", 2.759f, 855},
    {2048, 2048, 0, 4, "rowmma.t8", 3.140f, 751},
    {2048, 2048, 0, 8, "rowmma.t8", 3.680f, 641},
    {8192, 8192, 0, 1, "rowlane", 11.215f, 3366},
    {8192, 8192, 0, 2, "rowlane", 12.262f, 3079},
    {8192, 8192, 0, 4, "rowmma.t8", 14.270f, 2645},
    {8192, 8192, 0, 8, "rowmma.t8", 21.730f, 1737},
    {2048, 1536, 0, 1, "rowlane", 2.056f, 861},
    {2048, 1536, 0, 2, "rowmma.t8", 2.580f, 686},
    {2048, 1536, 0, 4, "rowmma.t8", 2.750f, 643},
    {2048, 1536, 0, 8, "rowmma.t8", 3.440f, 514},
    {2048, 6144, 1, 1, "rowlane", 4.712f, 3004},
    {2048, 6144, 1, 2, "rowlane", 6.038f, 2344},
    {2048, 6144, 1, 4, "rowmma.t8c2", 7.380f, 1918},
    {2048, 6144, 1, 8, "rowmma.t8c2", 8.590f, 1648},
    {6144, 2048, 0, 1, "rowlane", 3.928f, 1802},
    {6144, 2048, 0, 2, "rowmma.t8", 4.090f, 1731},
    {6144, 2048, 0, 4, "rowmma.t8", 4.490f, 1576},
    {6144, 2048, 0, 8, "rowmma.t8", 5.500f, 1287},
    {4096, 11008, 1, 1, "rowlane", 10.908f, 4650},
    {4096, 11008, 1, 2, "rowlane", 13.192f, 3845},
    {4096, 11008, 1, 4, "rowmma.t8", 18.380f, 2760},
    {4096, 11008, 1, 8, "rowmma.t8", 21.570f, 2352},
    {11008, 4096, 0, 1, "rowmma", 8.008f, 3167},
    {11008, 4096, 0, 2, "rowlane", 9.796f, 2589},
    {11008, 4096, 0, 4, "rowmma.t8", 11.630f, 2181},
    {11008, 4096, 0, 8, "rowmma.t8", 13.750f, 1845},
    {5120, 5120, 0, 1, "rowlane", 4.912f, 3002},
    {5120, 5120, 0, 2, "rowlane", 6.379f, 2312},
    {5120, 5120, 0, 4, "rowmma.t8", 7.550f, 1953},
    {5120, 5120, 0, 8, "rowmma.t8", 8.770f, 1681},
    {5120, 27648, 1, 1, "l8r1u2w4", 33.920f, 4695},
    {5120, 27648, 1, 2, "l8r1u2w4", 40.944f, 3890},
    {5120, 27648, 1, 4, "l8r1u2w4", 60.360f, 2638},
    {5120, 27648, 1, 8, "rowmma.t8", 100.950f, 1578},
    {27648, 5120, 0, 1, "rowlane", 20.390f, 3905},
    {27648, 5120, 0, 2, "rowlane", 24.013f, 3316},
    {27648, 5120, 0, 4, "rowlane", 34.688f, 2295},
    {27648, 5120, 0, 8, "rowlane", 34.515f, 2307},
};
constexpr int kMeasuredRankCount = static_cast<int>(sizeof(kMeasuredRanks) / sizeof(kMeasuredRanks[0]));

}  // namespace vecq
}  // namespace llmp_b200

#endif  // LLMP_B200_CSRC_VECQ_RANKS_H_
