// Instantiations of the tiled FP64 M2L, orders 2..6.
#include <algorithm>

#include "m2l_tile_kernel.cuh"

namespace sfmm {
namespace tile {

bool launch_lo(const EvalArgs& a, const TileArgs& g, int warps, int sms, cudaStream_t st)
{
    switch (a.p) {
    case 2: return launch_p<2>(a, g, warps, sms, st);
    case 3: return launch_p<3>(a, g, warps, sms, st);
    case 4: return launch_p<4>(a, g, warps, sms, st);
    case 5: return launch_p<5>(a, g, warps, sms, st);
    case 6: return launch_p<6>(a, g, warps, sms, st);
    default: return false;
    }
}

}  // namespace tile
}  // namespace sfmm
