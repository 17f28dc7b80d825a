// Stage-kernel instantiations of the FP32-mixed form.
#include "kernel_table.cuh"

namespace mhdb {

namespace {
using Cfg0 = TileCfg<32, 16, 256, 2>; // default
using Cfg1 = TileCfg<32, 16, 256, 3>;
using Cfg2 = TileCfg<32, 8, 256, 3>;
using Cfg3 = TileCfg<32, 16, 384, 2, true>;
using Cfg4 = TileCfg<32, 16, 256, 2, true>;
using Cfg5 = TileCfg<32, 8, 320, 3, true>;
using Cfg6 = MarchCfg<4, 64, 3>;
using Cfg7 = MarchTmaCfg<4, 32, 4>;
using Cfg8 = MarchTmaCfg<2, 32, 8>;
using Cfg9 = MarchTmaCfg<1, 32, 16>;
using Cfg10 = MarchTmaCfg<4, 32, 4, true, 0>;
using Cfg11 = MarchTmaCfg<1, 32, 16, true, 0>;
using Cfg12 = MarchTmaCfg<1, 64, 16>;
using Cfg13 = MarchTmaCfg<1, 32, 16, true, 0, 0, 1>; // increment form (also masked)
using Cfg14 = MarchTmaCfg<1, 64, 16, true, 0, 0, 1>; // increment form, 64-row segments
using Cfg15 = MarchPairCfg<32, 8>;  // increment form, two columns per lane
using Cfg16 = MarchPairCfg<32, 10>; // the same, 10 blocks per SM requested (168 registers)
// increment form, stage 2's own-cell delta from the halo stream (also masked)
using Cfg17 = MarchTmaCfg<1, 32, 16, true, 0, 0, 2>;
using Cfg18 = MarchCfg<1, 32, 16>; // one-warp register march (stored form)
constexpr TileConfigInfo kInfo[] = {
    {32, 16, 256, 2, kKindTile},       {32, 16, 256, 3, kKindTile},
    {32, 8, 256, 3, kKindTile},        {32, 16, 384, 2, kKindTileMerged},
    {32, 16, 256, 2, kKindTileMerged}, {32, 8, 320, 3, kKindTileMerged},
    {112, 64, 128, 3, kKindMarch},     {112, 32, 128, 4, kKindMarchTma},
    {56, 32, 64, 8, kKindMarchTma},    {28, 32, 32, 16, kKindMarchTma},
    {112, 32, 128, 4, kKindMarchTma},  {28, 32, 32, 16, kKindMarchTma},
    {28, 64, 32, 16, kKindMarchTma},   {28, 32, 32, 16, kKindMarchTmaDelta},
    {28, 64, 32, 16, kKindMarchTmaDelta}, {60, 32, 32, 8, kKindMarchTmaPair},
    {60, 32, 32, 10, kKindMarchTmaPair}, {28, 32, 32, 16, kKindMarchTmaDelta},
    {28, 32, 32, 16, kKindMarch}};
constexpr int kCount = sizeof(kInfo) / sizeof(kInfo[0]);
} // namespace

int stage_config_count_mixed() { return kCount; }

// Without a chosen configuration: unmasked grids of at least 1024^2 cells run the TMA strip march of
// the increment form with stage 2's own-cell increment taken from the halo stream (configuration
// 17); smaller ones the one-warp register march of the stored form (configuration 18), which has no
// copies to set up (per step, register against TMA march: 128^2 13.7 and 15.2 us, 301x173 17.1 and
// 19.2, 400^2 26.6 and 29.6, 512^2 38 and 40, 640^2 49 and 50, 724^2 56 and 56; the tile kernel took
// 18.5, 21.5, 36, 46 and 168 us at 128^2, 301x173, 400^2, 512^2 and 1024^2). From 724^2 up the TMA
// march is the faster one (900^2 90 and 84 us, 1024^2 110 and 99), but the increment form's stage 2
// reads U* as fl(hi(U^n) + delta), rounded twice where the stored hi plane is rounded once, and its
// error against FP64 is 10 to 16 % larger (800x760: 2.9e-8 against 2.6e-8), so it serves only the
// sizes it was chosen for.
// Masked grids of at least 1024^2 cells run the stored-form TMA march (configuration 11), smaller
// ones the tile kernel: the march stores a solid cell from the row's FP32 primitives, the tile kernel
// from the FP64 wall fill, so the march stays with the sizes it was chosen for (512^2 74 against 68
// us, 724^2 102 against 117).
int default_stage_config_mixed(long long cells, bool mask)
{
    if (mask) {
        return cells >= 1024LL * 1024 ? 11 : 0;
    }
    return cells >= 1024LL * 1024 ? 17 : 18;
}

TileConfigInfo stage_config_info_mixed(int c) { return kInfo[c < 0 || c >= kCount ? 0 : c]; }

StageKernels select_stage_mixed(int limiter, bool nonideal, bool mask, int config)
{
    switch (config) {
    case 1:
        return select_unmasked<PolicyMixed, Cfg1>(limiter, nonideal, mask);
    case 2:
        return select_unmasked<PolicyMixed, Cfg2>(limiter, nonideal, mask);
    case 3:
        return select_unmasked<PolicyMixed, Cfg3>(limiter, nonideal, mask);
    case 4:
        return select_unmasked<PolicyMixed, Cfg4>(limiter, nonideal, mask);
    case 5:
        return select_unmasked<PolicyMixed, Cfg5>(limiter, nonideal, mask);
    case 6:
        return select_unmasked<PolicyMixed, Cfg6>(limiter, nonideal, mask);
    case 7:
        return select_unmasked<PolicyMixed, Cfg7>(limiter, nonideal, mask);
    case 8:
        return select_unmasked<PolicyMixed, Cfg8>(limiter, nonideal, mask);
    case 9:
        return select_unmasked<PolicyMixed, Cfg9>(limiter, nonideal, mask);
    case 10:
        return select_unmasked<PolicyMixed, Cfg10>(limiter, nonideal, mask);
    case 11:
        return select_full<PolicyMixed, Cfg11>(limiter, nonideal, mask);
    case 12:
        return select_unmasked<PolicyMixed, Cfg12>(limiter, nonideal, mask);
    case 13:
        return select_full<PolicyMixed, Cfg13>(limiter, nonideal, mask);
    case 14:
        return select_unmasked<PolicyMixed, Cfg14>(limiter, nonideal, mask);
    case 15:
        return select_unmasked<PolicyMixed, Cfg15>(limiter, nonideal, mask);
    case 16:
        return select_unmasked<PolicyMixed, Cfg16>(limiter, nonideal, mask);
    case 17:
        return select_full<PolicyMixed, Cfg17>(limiter, nonideal, mask);
    case 18:
        return select_unmasked<PolicyMixed, Cfg18>(limiter, nonideal, mask);
    default:
        return select_full<PolicyMixed, Cfg0>(limiter, nonideal, mask);
    }
}

} // namespace mhdb
