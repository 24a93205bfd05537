// tile_parts.h: sizes of the tiled M2L's part sums and what a server sets aside.
#include <cstdio>

#include "tile_parts.h"

#define CHECK(c) do { if (!(c)) { std::printf("line %d: %s\n", __LINE__, #c); return 1; } } while (0)

int main()
{
    using namespace sfmm;
    // p = 10: 6 parts x (2 x 66 + 78) complex values a row
    CHECK(tile_part_bytes(1, 10) == 6 * 210 * 16);
    // coarse sizes: at least the size, at most an eighth more, multiples of 16, the same for sizes a percent apart mostly
    size_t last = 0;
    for (size_t b = 16; b < (size_t(1) << 40); b += b / 7 + 16) {
        const size_t c = coarse_bytes(b);
        CHECK(c >= b && c % 16 == 0 && (c - b) * 8 <= b + 128 && c >= last && coarse_bytes(c) == c);
        last = c;
    }
    CHECK(coarse_bytes(tile_part_bytes(18615, 10)) == coarse_bytes(tile_part_bytes(18500, 10)));
    // measured node counts (levels >= 2) are covered: points, leaf size, nodes
    const long got[][3] = {{300007, 64, 18615}, {370000, 64, 22643}, {20000, 64, 1341}, {60000, 64, 4681}, {40000, 64, 4449}};
    for (auto& g : got)
        for (int p = 2; p <= 12; ++p) CHECK(tile_part_estimate(g[0], int(g[1]), 1, p) >= tile_part_bytes(g[2], p));
    // vector charges of a uniform cloud: 210,000 points are about 5,200 nodes, 15,600 rows
    CHECK(tile_part_estimate(215000, 64, 3, 10) >= tile_part_bytes(3 * 5209, 10));
    // never more than a plan can take; none for trees that are surely too large or orders without parts
    for (int n = 1000; n < 4000000; n += n / 9)
        for (int q = 1; q <= 3; ++q) CHECK(tile_part_estimate(n, 64, q, 12) <= coarse_bytes(tile_part_bytes(kTileSplitRows, 12)));
    CHECK(tile_part_estimate(4000000, 64, 1, 10) == 0 && tile_part_estimate(20000, 64, 1, 13) == 0 && tile_part_estimate(20000, 64, 1, 1) == 0);
    CHECK(tile_part_estimate(1, 1, 1, 2) > 0 && tile_part_estimate(1000, 0, 1, 2) > 0);
    std::printf("tile parts ok\n");
    return 0;
}
