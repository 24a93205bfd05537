// FP64 M2L (fmm.hpp:620-688) for orders 2..12: rotate, translate along z,
// rotate back, as FP64 tensor-core products (mma.sync m8n8k4 f64) over tiles of
// targets that share every offset.
//
// Work decomposition.  All targets of one octant (position in the parent) at
// one level have their sources at the same offsets d, so for a given d they
// share the whole operator: rotation class, distance and azimuth.  A warp owns
// 8 columns (the N of the MMA; a column is a target and a charge component):
// children in one octant of consecutive split parents of a level.  The block's
// warps run over the same slots (the offsets that occur, at most 189 of the
// 6 x 6 x 6 box around the target) with one copy of the slot's operators; a
// target without a source in a slot takes zero moments.  Large trees order a
// level's parents by which of their 27 neighbours are split, so that a block's
// targets have the same slots.
//
// Per slot, with expansions of the level scaled by the box size w
// (M~_n = w^-n M_n, L_j = w^-(j+1) L~_j; the factor w^-n rides on the phases):
//   R  X = e^{i m phi} M~ (formed as operands are read), W_n = (P_n Re X_n,
//      Q_n Im X_n) for orders n < p
//   T  Lz^k = T_k W^k, the distance in the operator, in place
//   I  L_j += e^{-i m phi} (PB_j Re Lz_j, QB_j Im Lz_j), orders j <= p + 1,
//      in registers over the slots of a part
// and after the slots a second pass D: the whole map (rotate, translate,
// rotate back) of the order-p moments, which the potential local (order p,
// sources <= p) has and the field local (order p + 1, sources < p) has not.
// The rest serves both.
//
// A warp's operands are its own, so its stages need no block barrier; the
// block shares only the operators.  These come by bulk copies, a buffer or two
// per stage (D: a ring of four), each with a full and an empty mbarrier; one
// warp per buffer refills it when every warp has left it.  All waits are
// bounded.  Operand buffers are laid out so that fragment loads and stores are
// free of bank conflicts.
//
// The sum over slots has a fixed association, whatever the block: six parts
// (the planes of one y offset, 36 slots each), added in part order.  One block
// runs all parts of its columns and adds each to LA / LB as it ends; or, for
// levels too small to fill the GPU so (kTileSplitRows), a block runs one part
// and k_tile_sum adds the parts in the same order.  No atomics.
//
// What bounds it: the FP64 unit, which DMMA (m8n8k4: 16 cycles a warp and
// sub-partition, latency 26) shares with DFMA, and the shared-memory operand
// reads between the MMAs; a slot of 8 warps takes about 14,000 cycles at
// p = 10, of which the unit is busy 8,400.  Three designs on the way, 4M Plummer
// points, p = 10: run-time job lists over 32 shared columns and three block
// barriers a slot 57 ms; the chunk loops unrolled 49 ms; a warp's own 8 columns
// 41 ms; loads moved before the stores they do not depend on and the ring for D
// 36.9 ms; in-place T and one refilling warp per buffer 35.7 ms.  (Per-warp
// straight-line code, 197 KB of it, missed the instruction cache: 114 ms.)
//
// Before (one block per sibling group, 8-column tiles of one class, an operator
// fragment load per MMA, five barriers per 8 columns: m2l.cu), 69.6 ms at that
// size, the FP64 unit 24% busy; 300k points p = 10 5.69 -> 3.42 ms; 400k p = 6
// potential 3.81 -> 2.21; 100k p = 8 1.19 -> 0.72; 2k p = 10 0.226 -> 0.185.
#include <cub/device/device_radix_sort.cuh>

#include <algorithm>
#include <cstdint>
#include <vector>

#include "m2l_tile.cuh"

namespace sfmm {
namespace {

using tile::imin;
using tile::up;

struct OpsArgs {
    const double* rot;
    const int* rot_off;
    int rot_len;
    const double* tzx;
    const int* tzx_off;
};

// Element (row, col) of fragment f of one class, P a run-time order (the
// layout of tile::Frags<P>).
__device__ double tile_entry(const OpsArgs& o, int P, int c, int f, int row, int col)
{
    const double* R = o.rot + int64_t(c) * o.rot_len;
    const double rho = sqrt(double(tile::class_dist2(c)));
    auto mat = [&](int n, int m, int r, int k) { return R[o.rot_off[n] + m * (n + 1) * (n + 1) + r * (n + 1) + k]; };
    // z-translation between scaled expansions: target order j, source order n, azimuth k
    auto tz = [&](int k, int j, int n) { return o.tzx[o.tzx_off[k] + (j - k) * (P + 1 - k) + (n - k)] * pow(rho, -double(j + n + 1)); };
    // rotation of orders n < P: per (row tile, K chunk) P then Q
    for (int n = 0; n < P; ++n) {
        const int KC = up(n + 1, 4), cnt = 2 * up(n + 1, 8) * KC;
        if (f < cnt) {
            const int r = 8 * (f / 2 / KC) + row, k = 4 * (f / 2 % KC) + col;
            if (r > n || k > n || ((f & 1) && (r == 0 || k == 0))) return 0.0;
            return mat(n, f & 1, r, k);
        }
        f -= cnt;
    }
    for (int k = 0; k < P; ++k) {
        const int KC = up(P - k, 4), cnt = up(P + 2 - k, 8) * KC;
        if (f < cnt) {
            const int j = k + 8 * (f / KC) + row, n = k + 4 * (f % KC) + col;
            return j <= P + 1 && n <= P - 1 ? tz(k, j, n) : 0.0;
        }
        f -= cnt;
    }
    for (int j = 0; j <= P + 1; ++j) {
        const int km = imin(j, P - 1), KP = up(km + 1, 4), KQ = up(km, 4), per = KP + KQ, cnt = up(j + 1, 8) * per;
        if (f < cnt) {
            const int r = 8 * (f / per) + row, h = f % per;
            const int q = h >= KP, k = q ? 1 + 4 * (h - KP) + col : 4 * h + col;
            if (r > j || k > km || (q && r == 0)) return 0.0;
            return mat(j, 2 + q, r, k);
        }
        f -= cnt;
    }
    // D: potential local row (j, m) from the order-P moments k
    const int T = (P + 1) * (P + 2) / 2, DK = up(P + 1, 4), dcnt = 2 * up(T, 8) * DK;
    if (f < dcnt) {
        const int r = 8 * (f / 2 / DK) + row, k = 4 * (f / 2 % DK) + col, q = f & 1;
        if (r >= T || k > P || (q && k == 0)) return 0.0;
        int j, m;
        tri_nm(r, j, m);
        if (q && m == 0) return 0.0;
        double v = 0.0;
        for (int b = q; b <= j; ++b) v += mat(j, 2 + q, m, b) * tz(b, j, P) * mat(P, q, b, k);
        return v;
    }
    return 0.0;
}

__global__ void k_tile_ops(OpsArgs o, int P, int per_class, double* __restrict__ out)
{
    const int64_t total = int64_t(tile::kClasses) * per_class * 32;
    for (int64_t e = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; e < total; e += int64_t(gridDim.x) * blockDim.x) {
        const int lane = static_cast<int>(e & 31), f = static_cast<int>((e >> 5) % per_class), c = static_cast<int>((e >> 5) / per_class);
        // class 7 t2i + dk + 3; (0, 0, dk) with |dk| <= 1 and other adjacent offsets never occur as sources
        out[e] = tile::class_dist2(c) > 0 ? tile_entry(o, P, c, f, lane >> 2, lane & 3) : 0.0;
    }
}

int frags_per_class(int P)
{
    int s = 0;
    for (int n = 0; n < P; ++n) s += 2 * up(n + 1, 8) * up(n + 1, 4);
    s += 2 * up((P + 1) * (P + 2) / 2, 8) * up(P + 1, 4);
    for (int k = 0; k < P; ++k) s += up(P + 2 - k, 8) * up(P - k, 4);
    for (int j = 0; j <= P + 1; ++j) s += up(j + 1, 8) * (up(imin(j, P - 1) + 1, 4) + up(imin(j, P - 1), 4));
    return s;
}

// Sort key of a split parent: its level, then which of its 27 neighbours are
// split (they hold its children's sources).
__global__ void k_tile_keys(const int32_t* __restrict__ list, int64_t n, const int64_t* __restrict__ lvl_off, int depth,
                            const int32_t* __restrict__ colleague, const int32_t* __restrict__ nchild, uint32_t* __restrict__ key)
{
    for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
        const int g = list[i];
        int l = 1;
        while (l < depth && g >= lvl_off[l + 1]) ++l;
        uint32_t m = 0;
        for (int s = 0; s < 27; ++s) {
            const int c = colleague[27 * int64_t(g) + s];
            if (c >= 0 && nchild[c] > 0) m |= 1u << s;
        }
        key[i] = uint32_t(l) << 27 | m;
    }
}

// Split tiles: the parts' sums scaled to the level and added in part order as
// the kernel does where one block has them all, a warp per target.
__global__ void k_tile_sum(EvalArgs a, tile::TileArgs g, int64_t chunks)
{
    const int lane = threadIdx.x & 31, qd = a.qdim;
    const int64_t stride = (int64_t(gridDim.x) * blockDim.x) >> 5, total = chunks * 8 * g.tpb;
    // the part sums of qd rows of `len` coefficients, then (more) the order-P sources'; lane j holds the scale of order j
    auto sum = [&](const cplx* part, const cplx* more, int64_t row, int len, double scale, cplx* out) {
        for (int e0 = 0; e0 < qd * len; e0 += 32) {
            const int e = e0 + lane;
            const bool on = e < qd * len;
            cplx w[2 * tile::kParts];
#pragma unroll
            for (int q = 0; q < 2 * tile::kParts; ++q) {
                if (q >= tile::kParts && !more) break;
                if (on) w[q] = (q < tile::kParts ? part : more)[((q % tile::kParts) * g.rows + row) * len + e];
            }
            int c = e, j, m;
            while (c >= len) c -= len;
            tri_nm(c, j, m);
            const double sc = __shfl_sync(0xffffffffu, scale, j);
            if (!on) continue;
            cplx v{0, 0};
#pragma unroll
            for (int q = 0; q < 2 * tile::kParts; ++q) {
                if (q >= tile::kParts && !more) break;
                v.re = fma(w[q].re, sc, v.re);
                v.im = fma(w[q].im, sc, v.im);
            }
            out[e] = v;
        }
    };
    for (int64_t w = (blockIdx.x * int64_t(blockDim.x) + threadIdx.x) >> 5; w < total; w += stride) {
        const int64_t cell = w / g.tpb;
        const int t = static_cast<int>(w % g.tpb), oct = static_cast<int>(cell & 7);
        const int4 ck = g.chunk[cell >> 3];
        if (t >= ck.y) continue;
        const int pr = g.parent[ck.x + t], cb = a.child_beg[pr], nc = a.nchild[pr];
        const double scale = pow(double(1 << ck.z) / a.box->width, double(lane + 1));
        int64_t node = -1;
        for (int k = 0; k < nc; ++k)
            if (static_cast<int>(a.key[cb + k] & 7) == oct) node = cb + k;
        if (node < 0) continue;
        const int64_t row = (node - g.node0) * qd;
        if (a.want_pot) sum(g.part_a, g.part_d, row, a.T, scale, a.LA + node * qd * a.T);
        if (a.want_field) sum(g.part_b, nullptr, row, a.T1, scale, a.LB + node * qd * a.T1);
    }
}

}  // namespace

void build_tile_ops(PlanTables& tb, int P, cudaStream_t st)
{
    const int nf = frags_per_class(P);
    tb.tile_ops.alloc(size_t(tile::kClasses) * nf * 32, st);
    tb.tile_zero.alloc(size_t(P + 1) * (P + 2), st);
    SFMM_CUDA(cudaMemsetAsync(tb.tile_zero.ptr, 0, tb.tile_zero.bytes(), st));
    OpsArgs o{tb.rot.ptr, tb.rot_off.ptr, tb.rot_len, tb.tzx.ptr, tb.tzx_off.ptr};
    k_tile_ops<<<512, 256, 0, st>>>(o, P, nf, tb.tile_ops.ptr);
    SFMM_CHECK_LAUNCH();
}

// Plans that run it: FP64 plans, and mixed plans whose M2L falls back to FP64
// (a shard, the rotation switch) below the order the TF32 kernel takes.
bool m2l_tile_supported(const Plan& pl)
{
    return pl.p >= kTileMinOrder && pl.p <= kTileMaxOrder && pl.tree->depth >= 2 && !pl.m2l_force_rows && !pl.i8 &&
           !(pl.precision == FMM_PRECISION_MIXED && pl.p >= kTf32MinOrder);
}

static thread_local size_t tl_part_limit = SIZE_MAX;

void set_thread_tile_part_limit(size_t bytes) noexcept { tl_part_limit = bytes; }

// Room for the part sums of `rows` rows; false (the parts then run in turn, to
// the same sums) where the thread's limit or the device has too little.
static bool take_parts(Plan& pl, int64_t rows)
{
    const size_t bytes = tile_part_bytes(rows, pl.p);
    if (rows >= kTileSplitRows || pl.m2l_whole_tiles || bytes > tl_part_limit) return false;
    try {
        pl.mt_part.alloc(std::min(coarse_bytes(bytes), tl_part_limit) / sizeof(double2), pl.tree->ctx->stream);
    } catch (const Error& e) {
        if (e.status != FMM_ERR_OUT_OF_MEMORY) throw;
        return false;
    }
    return true;
}

// Chunks of at most pl.mt_tpb parents [b, e) per level.
static void tile_chunks(Plan& pl, Plan::TileList& tl, const std::vector<int32_t>& b, const std::vector<int32_t>& e)
{
    std::vector<int4> ck;
    for (int q = 1; q < pl.tree->depth; ++q)
        for (int32_t s = b[q]; s < e[q]; s += pl.mt_tpb) ck.push_back(make_int4(s, imin(pl.mt_tpb, e[q] - s), q + 1, 0));
    tl.chunks = static_cast<int64_t>(ck.size());
    if (ck.empty()) return;
    cudaStream_t st = pl.tree->ctx->stream;
    tl.chunk.alloc(ck.size(), st);
    SFMM_CUDA(cudaMemcpyAsync(tl.chunk.ptr, ck.data(), ck.size() * sizeof(int4), cudaMemcpyHostToDevice, st));
}

// Tiles of the plan's tree.  pl.sh_list / pl.sh_S hold the split parents level
// by level.
void m2l_tile_setup(Plan& pl)
{
    pl.mt_all.chunks = 0;
    pl.mt_groups = 0;
    pl.mt_on = false;
    if (!m2l_tile_supported(pl)) return;
    Tree& t = *pl.tree;
    // sparse lists take the group kernel; a forest decides member by member, so that a member's result does not
    // depend on its company
    const bool forest = !t.member_sparse.empty();
    bool some = forest ? false : m2l_sparse(t.il_nnz, t.n_nodes - t.lvl_off[2]), all = some;
    if (forest) {
        all = true;
        for (uint8_t v : t.member_sparse) {
            some |= v != 0;
            all &= v != 0;
        }
    }
    if (all) return;
    pl.mt_on = true;
    cudaStream_t st = t.ctx->stream;
    const int sms = t.ctx->sm_count;
    const int64_t n = pl.sh_S[t.depth];
    if (n == 0) return;
    // few targets: the parts of a tile in blocks of their own, and if that does not give every SM two full blocks to
    // run one after the other, narrow tiles (p = 10 at one, two and four blocks, M2L: Plummer 100k points 1.35, 1.35
    // and 1.92 ms; p = 6, 60k 0.57, 0.46 and 0.46 ms).  From order 11 on one narrow block's operators
    // fill an SM (119 KB of shared memory), two warps, and full blocks are faster: M2L at p = 12, narrow and full, of
    // Plummer 20k points 1.56 and 1.13 ms, 10k in leaves of 32 1.43 and 0.98; whole evaluations of 41 small trees,
    // full / narrow in the mean 0.80 at p = 11 and 0.84 at 12 (0.61 to 1.04), but 1.14 at 6, 1.13 at 8, 1.03 at 10
    const int64_t rows = (t.lvl_off[t.depth + 1] - t.lvl_off[2]) * pl.qdim;
    const int full = tile::full_warps(pl.p);
    pl.mt_split = take_parts(pl, rows);
    pl.mt_warps = pl.mt_split && pl.p <= tile::kNarrowMaxOrder && rows * tile::kParts < int64_t(sms) * 2 * 8 * full ? tile::kSmallWarps : full;
    pl.mt_tpb = 8 * pl.mt_warps / pl.qdim;
    std::vector<int32_t> b(pl.sh_S), e(pl.sh_S);             // per level: parents [b, e)
    for (int q = 1; q < t.depth; ++q) e[q] = pl.sh_S[q + 1];
    pl.mt_all.parent.alloc(n, st);
    if (some) {
        // the forest's split parents, those of sparse members apart
        std::vector<int32_t> list(n), tiled, group;
        SFMM_CUDA(cudaMemcpyAsync(list.data(), pl.sh_list.ptr, n * sizeof(int32_t), cudaMemcpyDeviceToHost, st));
        SFMM_CUDA(cudaStreamSynchronize(st));
        const size_t B = t.member_sparse.size();
        for (int q = 1; q < t.depth; ++q) {
            const auto first = t.member_node.begin() + q * (B + 1);
            b[q] = static_cast<int32_t>(tiled.size());
            for (int32_t i = pl.sh_S[q]; i < pl.sh_S[q + 1]; ++i) {
                const size_t r = std::upper_bound(first, first + B + 1, int64_t(list[i])) - first - 1;
                (t.member_sparse[r] ? group : tiled).push_back(list[i]);
            }
            e[q] = static_cast<int32_t>(tiled.size());
        }
        pl.mt_groups = static_cast<int64_t>(group.size());
        pl.mt_group.alloc(std::max<size_t>(group.size(), 1), st);
        if (!group.empty())
            SFMM_CUDA(cudaMemcpyAsync(pl.mt_group.ptr, group.data(), group.size() * sizeof(int32_t), cudaMemcpyHostToDevice, st));
        if (!tiled.empty())
            SFMM_CUDA(cudaMemcpyAsync(pl.mt_all.parent.ptr, tiled.data(), tiled.size() * sizeof(int32_t), cudaMemcpyHostToDevice, st));
        SFMM_CUDA(cudaStreamSynchronize(st));
    }
    if (!some && n >= kTileSortMin) {
        DevBuf<uint32_t> k0, k1;
        DevBuf<int64_t> lvl;
        k0.alloc(n, st);
        k1.alloc(n, st);
        lvl.alloc(t.lvl_off.size(), st);
        SFMM_CUDA(cudaMemcpyAsync(lvl.ptr, t.lvl_off.data(), t.lvl_off.size() * sizeof(int64_t), cudaMemcpyHostToDevice, st));
        k_tile_keys<<<blocks_for(n, 256, int64_t(sms) * 8), 256, 0, st>>>(pl.sh_list.ptr, n, lvl.ptr, t.depth, t.colleague.ptr,
                                                                         t.nchild.ptr, k0.ptr);
        SFMM_CHECK_LAUNCH();
        size_t tmp_bytes = 0;
        SFMM_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tmp_bytes, k0.ptr, k1.ptr, pl.sh_list.ptr, pl.mt_all.parent.ptr,
                                                  static_cast<int>(n), 0, 32, st));
        DevBuf<uint8_t> tmp;
        tmp.alloc(std::max<size_t>(tmp_bytes, 1), st);
        SFMM_CUDA(cub::DeviceRadixSort::SortPairs(tmp.ptr, tmp_bytes, k0.ptr, k1.ptr, pl.sh_list.ptr, pl.mt_all.parent.ptr,
                                                  static_cast<int>(n), 0, 32, st));
    } else if (!some) {
        SFMM_CUDA(cudaMemcpyAsync(pl.mt_all.parent.ptr, pl.sh_list.ptr, n * sizeof(int32_t), cudaMemcpyDeviceToDevice, st));
    }
    tile_chunks(pl, pl.mt_all, b, e);
    if (pl.mt_all.chunks == 0) return;
    const int64_t items = pl.mt_all.chunks * 8 * (pl.mt_split ? tile::kParts : 1);
    const int64_t blocks = std::min<int64_t>(items, int64_t(sms) * tile::max_per_sm(pl.mt_warps));
    pl.mt_table.alloc(coarse_bytes(size_t(blocks) * 2 * tile::kSlots * 8 * pl.mt_warps * sizeof(int32_t)) / sizeof(int32_t), st);
}

// Tiles of the shard's parents, beside the whole tree's (a captured graph
// launches on those); slot tables, part sums and widths are the tree's.
void m2l_tile_shard(Plan& pl)
{
    Tree& t = *pl.tree;
    pl.mt_shard.chunks = 0;
    const int64_t n = pl.mt_on ? pl.sh_S[t.depth] : 0;
    if (n == 0) return;
    cudaStream_t st = t.ctx->stream;
    std::vector<int32_t> list(n), b(t.depth), e(t.depth);
    SFMM_CUDA(cudaMemcpyAsync(list.data(), pl.sh_list.ptr, n * sizeof(int32_t), cudaMemcpyDeviceToHost, st));
    SFMM_CUDA(cudaStreamSynchronize(st));
    for (int q = 1; q < t.depth; ++q) {
        const auto lo = list.begin() + pl.sh_S[q], hi = list.begin() + pl.sh_S[q + 1];
        b[q] = static_cast<int32_t>(std::lower_bound(lo, hi, pl.own_parent_b[q]) - list.begin());
        e[q] = static_cast<int32_t>(std::lower_bound(lo, hi, pl.own_parent_e[q]) - list.begin());
    }
    pl.mt_shard.parent.alloc(n, st);
    SFMM_CUDA(cudaMemcpyAsync(pl.mt_shard.parent.ptr, pl.sh_list.ptr, n * sizeof(int32_t), cudaMemcpyDeviceToDevice, st));
    tile_chunks(pl, pl.mt_shard, b, e);
}

bool launch_m2l_tile(Plan& pl, const EvalArgs& a, cudaStream_t st)
{
    if (!pl.mt_on || !m2l_tile_supported(pl)) return false;
    const Tree& t = *pl.tree;
    const int sms = t.ctx->sm_count;
    if (pl.mt_groups > 0) {
        EvalArgs b = a;
        b.m2l_list = pl.mt_group.ptr;
        launch_m2l(b, 0, pl.mt_groups, sms, st);
    }
    const Plan::TileList& tl = pl.shard_count > 1 ? pl.mt_shard : pl.mt_all;
    if (tl.chunks == 0) return true;                         // no (other) targets
    tile::TileArgs g{};
    g.ops = pl.tab->tile_ops.ptr;
    g.parent = tl.parent.ptr;
    g.chunk = tl.chunk.ptr;
    g.items = tl.chunks * 8 * (pl.mt_split ? tile::kParts : 1);
    g.tpb = pl.mt_tpb;
    g.split = pl.mt_split;
    g.node0 = t.lvl_off[2];
    g.rows = (t.lvl_off[t.depth + 1] - t.lvl_off[2]) * pl.qdim;
    g.part_a = reinterpret_cast<cplx*>(pl.mt_part.ptr);
    g.part_d = g.part_a + tile::kParts * g.rows * pl.T;
    g.part_b = g.part_d + tile::kParts * g.rows * pl.T;
    g.table = pl.mt_table.ptr;
    g.zero = reinterpret_cast<const cplx*>(pl.tab->tile_zero.ptr);
    g.ctr = pl.m2l_ctr.ptr;
    const bool done = a.p <= 6   ? tile::launch_lo(a, g, pl.mt_warps, sms, st)
                      : a.p <= 9 ? tile::launch_mid(a, g, pl.mt_warps, sms, st)
                                 : tile::launch_hi(a, g, pl.mt_warps, sms, st);
    if (done && pl.mt_split) {
        k_tile_sum<<<blocks_for(tl.chunks * 8 * pl.mt_tpb * 32, 256, int64_t(sms) * 16), 256, 0, st>>>(a, g, tl.chunks);
        SFMM_CHECK_LAUNCH();
    }
    return done;
}

}  // namespace sfmm
