// Instantiations of the tiled FP64 M2L, orders 10..12.
#include <algorithm>

#include "m2l_tile_kernel.cuh"

namespace sfmm {
namespace tile {

bool launch_hi(const EvalArgs& a, const TileArgs& g, int warps, int sms, cudaStream_t st)
{
    switch (a.p) {
    case 10: return launch_p<10>(a, g, warps, sms, st);
    case 11: return launch_p<11>(a, g, warps, sms, st);
    case 12: return launch_p<12>(a, g, warps, sms, st);
    default: return false;
    }
}

}  // namespace tile
}  // namespace sfmm
