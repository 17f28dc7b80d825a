// Stage-kernel instantiations of the plain FP64 form.
#include "kernel_table.cuh"

namespace mhdb {

namespace {
using Cfg0 = TileCfg<32, 8, 256, 2>; // default
using Cfg1 = TileCfg<32, 4, 128, 4>;
using Cfg2 = TileCfg<32, 8, 320, 2>;
using Cfg3 = TileCfg<32, 8, 320, 2, true>;
using Cfg4 = MarchCfg<4, 64, 2>;
using Cfg5 = MarchCfg<4, 64, 3>;
using Cfg6 = MarchTmaCfg<1, 32, 8, true, 0, 0>;
using Cfg7 = MarchTmaCfg<1, 32, 10, true, 0, 0>;
using Cfg8 = MarchCfg<1, 32, 12>; // rows loaded by the lanes: any row pitch and base alignment
constexpr TileConfigInfo kInfo[] = {{32, 8, 256, 2, kKindTile},    {32, 4, 128, 4, kKindTile},
                                    {32, 8, 320, 2, kKindTile},    {32, 8, 320, 2, kKindTileMerged},
                                    {112, 64, 128, 2, kKindMarch}, {112, 64, 128, 3, kKindMarch},
                                    {28, 32, 32, 8, kKindMarchTma}, {28, 32, 32, 10, kKindMarchTma},
                                    {28, 32, 32, 12, kKindMarch}};
constexpr int kCount = sizeof(kInfo) / sizeof(kInfo[0]);
} // namespace

int stage_config_count_f64() { return kCount; }

// Without a chosen configuration: unmasked FP64 grids run a strip march, whose segments are cut to
// the grid (segment_rows): below 448^2 cells, where the state stays in L2 and a stage is a chain of
// latencies, the one-warp register march (configuration 8), above the TMA march (configuration 7).
// Per step, tile kernel (configuration 2) / register / TMA march: 128^2 15.8 / 14.0 / 15.1 us, 256^2
// 23.3 / 24.1 / 25.7, 300x173 23.7 / 20.9 / 21.4, 400^2 48.9 / 37.9 / 38.6, 512^2 67 / 52.4 / 51.1,
// 1024^2 258 / 204 / 162 (at 256^2 the tile kernel's blocks fill exactly one wave). Masked grids
// march from 1200^2 cells up and run the tile kernel (configuration 0) below: 512^2 83 against 105
// us, 1024^2 304 and 313, 1448^2 594 and 506.
int default_stage_config_f64(long long cells, bool mask)
{
    if (mask) {
        return cells >= 1200LL * 1200 ? 7 : 0;
    }
    return cells >= 448LL * 448 ? 7 : 8;
}

TileConfigInfo stage_config_info_f64(int c) { return kInfo[c < 0 || c >= kCount ? 0 : c]; }

StageKernels select_stage_f64(int limiter, bool nonideal, bool mask, int config)
{
    switch (config) {
    case 1:
        return select_unmasked<PolicyF64, Cfg1>(limiter, nonideal, mask);
    case 2:
        return select_unmasked<PolicyF64, Cfg2>(limiter, nonideal, mask);
    case 3:
        return select_unmasked<PolicyF64, Cfg3>(limiter, nonideal, mask);
    case 4:
        return select_unmasked<PolicyF64, Cfg4>(limiter, nonideal, mask);
    case 5:
        return select_unmasked<PolicyF64, Cfg5>(limiter, nonideal, mask);
    case 6:
        return select_unmasked<PolicyF64, Cfg6>(limiter, nonideal, mask);
    case 8:
        return select_unmasked<PolicyF64, Cfg8>(limiter, nonideal, mask);
    case 7:
        return select_full<PolicyF64, Cfg7>(limiter, nonideal, mask);
    default:
        return select_full<PolicyF64, Cfg0>(limiter, nonideal, mask);
    }
}

} // namespace mhdb
