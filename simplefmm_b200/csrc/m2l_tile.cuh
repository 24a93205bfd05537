// FP64 M2L on the FP64 tensor cores over tiles of targets that share every
// offset (orders 2..12): declarations shared by the kernel's instantiations
// (m2l_tile_*.cu) and its host side (m2l_tile.cu).
#pragma once

#include <type_traits>

#include "eval_util.cuh"

namespace sfmm {
namespace tile {

constexpr int kSlots = 216;               // offsets of an octant: a 6 x 6 x 6 box around the target
constexpr int kClasses = 70;              // rotation classes (fmm.hpp:169)
constexpr int kParts = kTileParts;        // parts of the slots: the planes of one y offset, 36 slots each
constexpr int kPartSlots = kSlots / kParts;
constexpr int kSmallWarps = 2;            // warps of a block when there are few tiles, orders up to kNarrowMaxOrder
constexpr int kNarrowMaxOrder = 10;

// |d|^2 of a rotation class (class = 7 t2i + dk + 3, fmm.hpp:171)
__host__ __device__ inline int class_dist2(int c)
{
    const int t2[10] = {0, 1, 2, 4, 5, 8, 9, 10, 13, 18};
    const int dk = c % 7 - 3;
    return t2[c / 7] + dk * dk;
}

__host__ __device__ constexpr int imin(int a, int b) { return a < b ? a : b; }
__host__ __device__ constexpr int up(int a, int b) { return (a + b - 1) / b; }

// Operator fragments (8 x 4 doubles, 256 bytes) of one class, by stage:
//   R  rotation of source orders n < P: per (n, row tile, K chunk) P then Q
//      (Q's m = 0 row and column are zero)
//   T  z-translation per azimuth k < P: rows j = k..P+1, sources n = k..P-1
//   I  inverse rotation per order j <= P+1: inputs k = 0..min(j, P-1) for the
//      real part, k = 1..min(j, P-1) for the imaginary part
//   D  per (row tile of the order-P potential local, K chunk) re then im: the
//      whole map (rotate, translate, rotate back) of the order-P moments
template<int P>
struct Frags {
    static constexpr int T = (P + 1) * (P + 2) / 2, T1 = (P + 2) * (P + 3) / 2;
    static constexpr int TW = P * (P + 1) / 2;              // coefficients of orders < P
    // Rows of the rotated / translated coefficients, azimuth by azimuth: azimuth k
    // has room for orders k..P+1, rounded up to 2 mod 4, so that the rows of one
    // order at consecutive azimuths lie 1 mod 4 apart (bank conflicts, see swz).
    __host__ __device__ static constexpr int az_rows(int k)
    {
        int n = P + 2 - k;
        while (n % 4 != 2) ++n;
        return n;
    }
    __host__ __device__ static constexpr int az(int k)
    {
        int s = 0;
        for (int i = 0; i < k; ++i) s += az_rows(i);
        return s;
    }
    static constexpr int ZI = up(az(P), 4) * 4;             // offset of the imaginary rows (4 | offset: the same swizzle)
    __host__ __device__ static constexpr int rt(int n) { return up(n + 1, 8); }
    __host__ __device__ static constexpr int kc(int n) { return up(n + 1, 4); }
    __host__ __device__ static constexpr int rot_off(int n)
    {
        int s = 0;
        for (int i = 0; i < n; ++i) s += 2 * rt(i) * kc(i);
        return s;
    }
    static constexpr int NR = rot_off(P);
    __host__ __device__ static constexpr int trt(int k) { return up(P + 2 - k, 8); }
    __host__ __device__ static constexpr int tkc(int k) { return up(P - k, 4); }
    __host__ __device__ static constexpr int tz_off(int k)
    {
        int s = 0;
        for (int i = 0; i < k; ++i) s += trt(i) * tkc(i);
        return s;
    }
    static constexpr int NT = tz_off(P);
    __host__ __device__ static constexpr int kmax(int j) { return imin(j, P - 1); }
    __host__ __device__ static constexpr int ikp(int j) { return up(kmax(j) + 1, 4); }
    __host__ __device__ static constexpr int ikq(int j) { return up(kmax(j), 4); }
    __host__ __device__ static constexpr int inv_off(int j)
    {
        int s = 0;
        for (int i = 0; i < j; ++i) s += rt(i) * (ikp(i) + ikq(i));
        return s;
    }
    static constexpr int NI = inv_off(P + 2);
    static constexpr int DT = up(T, 8), DK = up(P + 1, 4), ND = 2 * DT * DK;
    static constexpr int per_class = NR + NT + NI + ND;     // in this order
    // row tiles whose sums a warp keeps in registers (8 registers each)
    __host__ __device__ static constexpr int inv_tiles(int j)
    {
        int s = 0;
        for (int i = 0; i < j; ++i) s += rt(i);
        return s;
    }
    static constexpr int IT = inv_tiles(P + 2);
};

// Warps of a full block: as many as the sums' registers (8 per row tile) and
// the operand buffers in shared memory leave room for.  At 255 registers some
// of it is still spilled: 76 bytes a thread at p = 10, 186 at 11, 266 at 8, 1,082
// at 12.
__host__ __device__ constexpr int full_warps(int P) { return P <= 6 ? 16 : P <= 8 ? 12 : P <= 10 ? 8 : 6; }

// resident blocks per SM at most (the blocks' slot tables are sized for them)
__host__ __device__ constexpr int max_per_sm(int warps) { return warps == kSmallWarps ? 4 : 1; }

struct TileArgs {
    const double* ops;                    // [class][per_class][32]
    const int32_t* parent;                // split parents, chunk by chunk
    const int4* chunk;                    // (first parent, parents, level of the targets, 0)
    int64_t items;                        // chunks x 8 octants (x kParts when split)
    int tpb;                              // targets per tile
    // split: an item is one part of a tile; its sums go, not yet scaled to the level, to part_a, part_b and part_d (the
    // order-P sources) [part][row], row = (node - node0) qdim + component, for k_tile_sum.  Else an item's parts are
    // scaled and added to the locals in part order, the same operations.
    int split;
    int64_t node0, rows;
    cplx *part_a, *part_b, *part_d;
    int32_t* table;                       // per block: [216][columns] source nodes, and the same warp by warp
    const cplx* zero;                     // a row of zero moments
    int* ctr;                             // counter the blocks take items from
};

// launch the kernel of order a.p with blocks of `warps` (kSmallWarps or
// full_warps); false: it does not fit the device
bool launch_lo(const EvalArgs& a, const TileArgs& g, int warps, int sms, cudaStream_t st);    // 2..6
bool launch_mid(const EvalArgs& a, const TileArgs& g, int warps, int sms, cudaStream_t st);   // 7..9
bool launch_hi(const EvalArgs& a, const TileArgs& g, int warps, int sms, cudaStream_t st);    // 10..12

}  // namespace tile
}  // namespace sfmm
