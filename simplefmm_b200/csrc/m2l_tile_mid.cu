// Instantiations of the tiled FP64 M2L, orders 7..9.
#include <algorithm>

#include "m2l_tile_kernel.cuh"

namespace sfmm {
namespace tile {

bool launch_mid(const EvalArgs& a, const TileArgs& g, int warps, int sms, cudaStream_t st)
{
    switch (a.p) {
    case 7: return launch_p<7>(a, g, warps, sms, st);
    case 8: return launch_p<8>(a, g, warps, sms, st);
    case 9: return launch_p<9>(a, g, warps, sms, st);
    default: return false;
    }
}

}  // namespace tile
}  // namespace sfmm
