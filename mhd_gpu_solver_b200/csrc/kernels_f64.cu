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

// Without a chosen configuration: unmasked FP64 grids run the TMA strip march (configuration 7),
// whose segments are cut to the grid (segment_rows), except where the tile kernel's blocks make
// one wave of two per SM and the march's just miss one, about 190^2 to 264^2 cells (per step at
// 256^2: tile 22.7, march 25.5 us; at 128^2 16.5 and 15.1, at 300^2 33 and 27, at 512^2 67 and 52,
// at 1024^2 258 and 163). There ideal solves take the 320-thread tile kernel (configuration 2),
// non-ideal ones configuration 0. Masked grids march from 2048^2 cells up and run configuration 0
// below (512^2 92 against 113 us, 1024^2 343 and 345, 2048^2 1294 and 1059).
int default_stage_config_f64(long long cells, bool mask, bool nonideal)
{
    if (mask) {
        return cells >= 2048LL * 2048 ? 7 : 0;
    }
    if (cells >= 190LL * 190 && cells < 264LL * 264) {
        return nonideal ? 0 : 2;
    }
    return 7;
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
