// The tiled FP64 M2L kernel (see m2l_tile.cu for the method).
#pragma once

#include "copy_parity.h"
#include "m2l_tile.cuh"

namespace sfmm {
namespace tile {

template<int B, int E, typename Fn>
__device__ __forceinline__ void static_for(Fn&& f)
{
    if constexpr (B < E) {
        f(std::integral_constant<int, B>{});
        static_for<B + 1, E>(f);
    }
}

// ------------------------------------------------------------------ PTX
__device__ __forceinline__ void dmma(double& d0, double& d1, double a, double b)
{
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};" : "+d"(d0), "+d"(d1) : "d"(a), "d"(b));
}
__device__ __forceinline__ uint32_t s32(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void bar_init(uint64_t* bar, int count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(s32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void bar_arrive(uint64_t* bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(s32(bar)) : "memory");
}
__device__ __forceinline__ void bar_expect(uint64_t* bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(s32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool bar_try(uint64_t* bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile("{\n.reg .pred q;\nmbarrier.try_wait.parity.shared::cta.b64 q, [%1], %2;\nselp.u32 %0, 1, 0, q;\n}\n"
                 : "=r"(ok)
                 : "r"(s32(bar)), "r"(parity)
                 : "memory");
    return ok != 0;
}
// Bounded wait of a warp: false when it expired or another warp gave up.
__device__ __forceinline__ bool bar_wait_long(uint64_t* bar, uint32_t parity, volatile int* abort)
{
    bool got = false;
    for (int it = 0; it < 1 << 22; ++it) {
        if (bar_try(bar, parity)) {
            got = true;
            break;
        }
        if ((it & 255) == 255 && *abort) break;
    }
    if (!got) *abort = 1;
    return __all_sync(0xffffffffu, got);
}
__device__ __forceinline__ bool bar_wait(uint64_t* bar, uint32_t parity, volatile int* abort)
{
    return __all_sync(0xffffffffu, bar_try(bar, parity)) || bar_wait_long(bar, parity, abort);
}
__device__ __forceinline__ void bulk(void* dst, const void* src, uint32_t bytes, uint64_t* bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(s32(dst)),
                 "l"(src), "r"(bytes), "r"(s32(bar))
                 : "memory");
}
__device__ __forceinline__ void proxy_fence() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// Shared-memory loads that the compiler may move past the stage's stores (they
// never touch the same rows, which it cannot see).  Their address must come
// from after(), which pins it behind the wait or warp barrier the data needs.
__device__ __forceinline__ uint32_t after(uint32_t addr)
{
    asm volatile("mov.b32 %0, %0;" : "+r"(addr)::"memory");
    return addr;
}
__device__ __forceinline__ double lds(uint32_t addr)
{
    double v;
    asm("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ double2 lds2(uint32_t addr)
{
    double2 v;
    asm("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(addr));
    return v;
}

// The loads that v depends on stay before this point.
__device__ __forceinline__ void before(double (&v)[4])
{
    asm volatile("" : "+d"(v[0]), "+d"(v[1]), "+d"(v[2]), "+d"(v[3])::"memory");
}

// ------------------------------------------------------------------ shared memory
// Per warp the slot's moments (written by bulk copies alone) and one buffer Z
// of rows of 8 columns that holds the rotated, then in place the translated
// coefficients.  Columns 4..7 and 0..3 of every other pair of rows are
// exchanged (swz): with the row offsets of Frags, fragment loads (4 rows x 8
// columns) and double2 stores (8 rows x 2 columns) are conflict free.
__device__ __forceinline__ int swz(int row) { return (row & 2) << 1; }
__host__ __device__ constexpr int pad4of8(int n) { return n + (12 - n % 8) % 8; }   // smallest >= n that is 4 mod 8

constexpr int kRing = 4;                  // D: operators and moments in flight
constexpr int kOps = 5;                   // operator buffers: R, T, T, I, I; or the D ring
constexpr int kDrainPolls = 1 << 16;      // of a barrier whose last copy is still in flight when the kernel gives up
template<int P, int NW>
struct Smem {
    using F = Frags<P>;
    static constexpr int CS = pad4of8(F::TW), CD = pad4of8(P + 1);   // column strides of the moments (complex)
    static constexpr int buf_m = up(16 * CS * 8, 128) * 128, buf_z = up(64 * 2 * F::ZI, 128) * 128;
    static constexpr int z = NW * buf_m;
    static constexpr int ops = z + NW * buf_z;              // R, T, I fragments; T and I twice where that fits
    static constexpr int DB = ops + 256 * (F::NR + 2 * F::NT + 2 * F::NI) + 8 * 1024 <= 227 * 1024 ? 2 : 1;
    static constexpr int ops_t = ops + 256 * F::NR, ops_i = ops_t + 256 * DB * F::NT;
    static constexpr int stages = ops_i + 256 * DB * F::NI;
    // D: rings of order-P moments per warp and of operators in the same space
    static constexpr int ring_m = 16 * CD * 8, ops_d = NW * kRing * ring_m;
    static constexpr int rings = ops_d + kRing * 256 * F::ND;
    static constexpr int lvl = stages > rings ? stages : rings;   // [P + 3] s^n of the level
    static constexpr int fsc = lvl + 8 * up(P + 3, 2) * 2;   // [P + 3] scales of the sums: s^n, or 1 (split: k_tile_sum scales)
    static constexpr int mask = fsc + 8 * up(P + 3, 2) * 2; // [216] x [NW] bytes: a warp's columns with a source
    static constexpr int used = mask + up(kSlots * NW, 16) * 16;   // [216] slots that occur
    static constexpr int cls = used + 4 * kSlots;           // [216] their rotation classes
    static constexpr int act = cls + up(kSlots, 16) * 16;           // [NW][216]: the warp's slots: index into used | slot << 8
    static constexpr int tgt = act + up(2 * kSlots * NW, 16) * 16; // [8 NW] target node of each tile position
    static constexpr int bars = tgt + 4 * 8 * NW;           // mbarriers: kRing per warp (moments); kOps operators full, empty
    static constexpr int misc = bars + 8 * (kRing * NW + 2 * kOps);   // item, slot count, abort
    static constexpr int total = misc + 16;
};

template<int P, int NW>
__global__ void __launch_bounds__(32 * NW, 1) k_m2l_tile(EvalArgs a, TileArgs g)
{
    using F = Frags<P>;
    using S = Smem<P, NW>;
    constexpr int T = F::T, T1 = F::T1, NC = 8 * NW, CS = S::CS, CD = S::CD, NTH = 32 * NW;
    extern __shared__ __align__(128) unsigned char sm[];
    double *lvl = reinterpret_cast<double*>(sm + S::lvl), *fsc = reinterpret_cast<double*>(sm + S::fsc);
    unsigned char* mask = sm + S::mask;
    int* used = reinterpret_cast<int*>(sm + S::used);
    unsigned char* cls = sm + S::cls;
    int* tgt = reinterpret_cast<int*>(sm + S::tgt);
    unsigned short* act = reinterpret_cast<unsigned short*>(sm + S::act) + (threadIdx.x >> 5) * kSlots;
    uint64_t* bars = reinterpret_cast<uint64_t*>(sm + S::bars);
    long long* item_s = reinterpret_cast<long long*>(sm + S::misc);
    int* ns_s = reinterpret_cast<int*>(sm + S::misc + 8);
    int* abort_s = reinterpret_cast<int*>(sm + S::misc + 12);
    volatile int* abort = abort_s;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, lr = lane >> 2, lc = lane & 3;
    const int qd = a.qdim, tpb = g.tpb;
    int32_t* table = g.table + int64_t(blockIdx.x) * 2 * kSlots * NC;
    int32_t* mine = table + kSlots * NC + (threadIdx.x >> 5) * kSlots * 8;   // the warp's sources, slot by slot
    // moments; operators (R, T, I or the D ring) landed; every warp done with them
    uint64_t *barM = bars + warp * kRing, *barO = bars + NW * kRing, *barE = barO + kOps;
    unsigned char *bufM = sm + warp * S::buf_m, *bufZ = sm + S::z + warp * S::buf_z;
    if (tid == 0) {
        for (int i = 0; i < kRing * NW + kOps; ++i) bar_init(bars + i, 1);
        for (int i = 0; i < kOps; ++i) bar_init(barE + i, NW);
        *abort_s = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    // parities of the next waits, a bit per barrier (barE: as barO); in parO, from bit kIssued on, of the operator copies
    // this thread issued to each (last_copy_parity; a warp's moments follow from its place in the pass, in_flight)
    uint32_t parM = 0, parO = 0;
    constexpr int kIssued = 16;

    for (;;) {
        if (tid == 0) *item_s = atomicAdd(g.ctr, 1);
        for (int s = tid; s < kSlots * NW; s += NTH) mask[s] = 0;
        __syncthreads();
        const int64_t item = *item_s;
        if (item >= g.items) break;
        const int64_t cell = g.split ? item / kParts : item;
        const int part0 = g.split ? static_cast<int>(item % kParts) : 0, part1 = g.split ? part0 + 1 : kParts;
        const int oct = static_cast<int>(cell & 7);
        const int cx = oct & 1, cy = (oct >> 1) & 1, cz = oct >> 2;
        const int4 ck = g.chunk[cell >> 3];
        const int lt = ck.z;
        // ---- set-up: the tile's targets, its sources per slot, the slots that occur
        for (int t = tid; t < NC; t += NTH) {
            int node = -1;
            if (t < ck.y) {
                const int pr = g.parent[ck.x + t];
                const int cb = a.child_beg[pr], nc = a.nchild[pr];
                for (int k = 0; k < nc; ++k)
                    if (static_cast<int>(a.key[cb + k] & 7) == oct) node = cb + k;
            }
            tgt[t] = node;
        }
        if (tid < P + 3) {
            lvl[tid] = pow(double(1 << lt) / a.box->width, double(tid));
            fsc[tid] = g.split ? 1.0 : lvl[tid];
        }
        __syncthreads();
        for (int t = warp; t < ck.y; t += NW) {
            const int node = tgt[t];
            if (node < 0) continue;
            for (int e = a.il_ptr[node] + lane; e < a.il_ptr[node + 1]; e += 32) {
                const int code = a.il_code[e], src = a.il_src[e];
                const int s = ((code >> 6) & 7) - 3 + 2 + cz + 6 * ((code & 7) - 3 + 2 + cx) + 36 * (((code >> 3) & 7) - 3 + 2 + cy);
                if (s / kPartSlots < part0 || s / kPartSlots >= part1) continue;
                for (int c = t * qd; c < (t + 1) * qd; ++c) {
                    table[s * NC + c] = src;
                    const int by = s * NW + (c >> 3);
                    atomicOr(reinterpret_cast<unsigned*>(mask + (by & ~3)), 1u << (8 * (by & 3) + (c & 7)));
                }
            }
        }
        __syncthreads();
        // rows of Z that are read before they are written (against zero operator entries) must be finite
        for (int e = tid; e < NW * S::buf_z / 16; e += NTH) reinterpret_cast<double2*>(sm + S::z)[e] = make_double2(0.0, 0.0);
        if (warp == 0) {
            int n = 0;
            for (int s0 = part0 * kPartSlots; s0 < part1 * kPartSlots; s0 += 32) {
                const int s = s0 + lane;
                bool on = false;
                if (s < part1 * kPartSlots)
                    for (int w = 0; w < NW; ++w) on |= mask[s * NW + w] != 0;
                const unsigned m = __ballot_sync(0xffffffffu, on);
                if (on) {
                    const int i = n + __popc(m & ((1u << lane) - 1u));
                    const int dz = s % 6 - 2 - cz, dx = (s / 6) % 6 - 2 - cx, dy = s / 36 - 2 - cy;
                    used[i] = s;
                    cls[i] = static_cast<unsigned char>(rot_class(dx, dy, dz));
                }
                n += __popc(m);
            }
            if (lane == 0) *ns_s = n;
        }
        __syncthreads();
        const int ns = *ns_s;
        int na = 0;                                         // the warp's slots: those in which it has a source
        for (int s0 = 0; s0 < ns; s0 += 32) {
            const bool on = s0 + lane < ns && mask[used[s0 + lane] * NW + warp] != 0;
            const unsigned m = __ballot_sync(0xffffffffu, on);
            if (on) act[na + __popc(m & ((1u << lane) - 1u))] = static_cast<unsigned short>((s0 + lane) | used[s0 + lane] << 8);
            na += __popc(m);
        }
        __syncwarp();
        for (int e = lane; e < na * 8; e += 32) {
            const int s = act[e >> 3] >> 8, c = e & 7;
            mine[e] = mask[s * NW + warp] >> c & 1 ? table[s * NC + warp * 8 + c] : -1;
        }
        __syncwarp();

        // source of lane's column (lanes 0..7) in the warp's k-th slot, -1: none
        const int bq = (warp * 8 + (lane & 7)) % qd;
        auto source = [&](int k) { return k < na && lane < 8 ? mine[k * 8 + lane] : -1; };
        // the moments (coefficients [first, first + count)) of those sources into b
        auto load_moments = [&](int src, unsigned char* b, int first, int count, int stride, int mb) {
            uint64_t* bar = barM + mb;
            if (lane == 0) bar_expect(bar, 8 * count * 16);
            __syncwarp();
            if (lane < 8)
                bulk(b + lane * stride * 16, src >= 0 ? a.M + (int64_t(src) * qd + bq) * T + first : g.zero, count * 16, bar);
        };
        auto load_ops = [&](int i, int first, int count, int where, int bar) {
            parO ^= 1u << (kIssued + bar);
            bar_expect(barO + bar, count * 256);
            bulk(sm + where, g.ops + (cls[i] * F::per_class + first) * 32, count * 256, barO + bar);
        };
        // the warp is done with operator buffer `bar`
        auto done = [&](int bar) {
            __syncwarp();
            if (lane == 0) bar_arrive(barE + bar);
        };
        // warp w, some time later: once every warp is done with buffer `bar` (parity of that use), load slot index
        // `to` into it
        auto reload = [&](int w, int bar, uint32_t parity, int to, int first, int count, int where) {
            if (warp != w % NW || to >= ns) return true;
            if (!bar_wait(barE + bar, parity, abort)) return false;
            if (lane == 0) load_ops(to, first, count, where, bar);
            return true;
        };
        // phases e^{i m phi} of slot s
        auto phases = [&](int s) {
            const int dx = (s / 6) % 6 - 2 - cx, dy = s / 36 - 2 - cy;
            return reinterpret_cast<const double2*>(a.eil) + (7 * (dy + 3) + dx + 3) * (P + 2);
        };
        bool ok = true;
        // local rows (node x component) of the lane's columns 2 lc, 2 lc + 1 (-1: no target)
        int64_t col_row[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int c = warp * 8 + 2 * lc + h, t = c / qd;
            const int node = t < tpb ? tgt[t] : -1;
            col_row[h] = node < 0 ? -1 : int64_t(node) * qd + (c - t * qd);
        }
        // ================ field local (and the potential local but for the order-P sources)
        {
            double sum[F::IT][4];                           // re, re, im, im of columns 2 lc, 2 lc + 1
#pragma unroll
            for (int u = 0; u < F::IT; ++u) sum[u][0] = sum[u][1] = sum[u][2] = sum[u][3] = 0.0;
            constexpr int DB = S::DB;
            // a part's sums, scaled back to the level, to the locals (or as they are to the part's own rows)
            bool fresh = true;
            auto flush = [&](int part) {
                const bool set = g.split || fresh;
                // both locals of a column; the rows' loads before the first store (kBatch in flight)
                constexpr int kBatch = 8;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int64_t row = col_row[h], pr = part * g.rows + row - g.node0 * qd;
                    if (row < 0) continue;
                    cplx* out_b = g.split ? g.part_b + pr * T1 : a.LB + row * T1;
                    cplx* out_a = g.split ? g.part_a + pr * T : a.LA + row * T;
                    static_for<0, 2 * up(F::IT, kBatch)>([&](auto bb) {
                        constexpr int first = decltype(bb)::value / 2 * kBatch, pot = decltype(bb)::value % 2;
                        if (!(pot ? a.want_pot : a.want_field)) return;
                        cplx* out = pot ? out_a : out_b;
                        cplx old[kBatch];
                        static_for<0, P + 2>([&](auto jj) {
                            constexpr int j = decltype(jj)::value;
                            if constexpr (j <= P + 1 - pot) {
#pragma unroll
                                for (int rt = 0; rt < F::rt(j); ++rt) {
                                    constexpr int u0 = F::inv_tiles(j);
                                    if (u0 + rt < first || u0 + rt >= first + kBatch) continue;
                                    const int m = 8 * rt + lr;
                                    old[u0 + rt - first] = !set && m <= j ? out[j * (j + 1) / 2 + m] : cplx{0, 0};
                                }
                            }
                        });
                        static_for<0, P + 2>([&](auto jj) {
                            constexpr int j = decltype(jj)::value;
                            if constexpr (j <= P + 1 - pot) {
                                const double sc = fsc[j + 1];
#pragma unroll
                                for (int rt = 0; rt < F::rt(j); ++rt) {
                                    constexpr int u0 = F::inv_tiles(j);
                                    if (u0 + rt < first || u0 + rt >= first + kBatch) continue;
                                    const int m = 8 * rt + lr;
                                    const double(&u)[4] = sum[u0 + rt];
                                    const cplx o = old[u0 + rt - first];
                                    if (m <= j) out[j * (j + 1) / 2 + m] = cplx{fma(u[h], sc, o.re), fma(u[2 + h], sc, o.im)};
                                }
                            }
                        });
                    });
                }
#pragma unroll
                for (int u = 0; u < F::IT; ++u) sum[u][0] = sum[u][1] = sum[u][2] = sum[u][3] = 0.0;
                fresh = false;
            };
            int k = 0;                                      // the warp's next slot
            if (na > 0) load_moments(source(0), bufM, 0, F::TW, CS, 0);
            int src = source(1);                            // sources of the slot after it
            if (ns > 0 && tid == 0) {
                load_ops(0, 0, F::NR, S::ops, 0);
                for (int u = 0; u < DB && u < ns; ++u) {
                    load_ops(u, F::NR, F::NT, S::ops_t + u * 256 * F::NT, 1 + u);
                    load_ops(u, F::NR + F::NT, F::NI, S::ops_i + u * 256 * F::NI, 3 + u);
                }
            }
            // Lane addresses in Z.  Loads: rows base + lc .. (columns lr); stores: rows base + lr (columns 2 lc,
            // 2 lc + 1); the swizzle depends on base % 4 alone.  A K chunk past the end of its order or azimuth reads
            // other rows of the same column (finite, against zero operator entries).
            int ld[4], st[4], rowk[up(P, 4)], rowq[up(P - 1, 4)], rowm[F::rt(P - 1)];
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                ld[b] = 8 * (lr ^ swz(lc + b));
                st[b] = 8 * ((2 * lc) ^ swz(lr + b));
            }
            auto azimuth = [&](int k) {                     // first row of azimuth k, less k
                int s = 0;
#pragma unroll
                for (int i = 0; i < P - 1; ++i) s += i < k ? F::az_rows(i) : 0;
                return 64 * (s - k);
            };
#pragma unroll
            for (int kc = 0; kc < up(P, 4); ++kc) rowk[kc] = azimuth(imin(4 * kc + lc, P - 1));
#pragma unroll
            for (int kc = 0; kc < up(P - 1, 4); ++kc) rowq[kc] = azimuth(imin(4 * kc + 1 + lc, P - 1));
#pragma unroll
            for (int rt = 0; rt < F::rt(P - 1); ++rt) rowm[rt] = azimuth(imin(8 * rt + lr, P - 1));
            const uint32_t m32 = s32(bufM) + 16 * (lr * CS + lc), z32 = s32(bufZ), ops32 = s32(sm + S::ops) + lane * 8;
            double2 e[up(P, 4)];                            // e^{i m phi} of the warp's next slot, m = 4 kc + lc
            int cur = na > 0 ? act[0] : 255;                // the warp's next slot (255: none; indices stay below)
            auto load_e = [&] {
                const double2* eil = phases(cur >> 8);
#pragma unroll
                for (int kc = 0; kc < up(P, 4); ++kc) e[kc] = __ldg(eil + imin(4 * kc + lc, P + 1));
            };
            if (na > 0) load_e();
            uint32_t parE = parO;                           // parities of the operators' earlier uses (T, I)
            bool counted = false;                           // given up with the k-th slot's moments counted as waited for
            for (int i = 0; i < ns; ++i) {
                const bool on = (cur & 255) == i;            // the warp has a source in this slot
                const int here = (cur >> 8) / kPartSlots;    // its part
                const int tb = 1 + i % DB, ib = 3 + i % DB;      // its T and I operator buffers
                double2 c[F::rt(P + 1)];                    // e^{i m phi}, m = 8 rt + lr
                // ---- R: X = e^{i m phi} s^n M, W_n = (P_n Re X_n, Q_n Im X_n)
                if (on) {
                    const double2* eil = phases(cur >> 8);
#pragma unroll
                    for (int rt = 0; rt < F::rt(P + 1); ++rt) c[rt] = __ldg(eil + imin(8 * rt + lr, P + 1));
                    ok = ok && bar_wait(barM, parM & 1u, abort);
                    parM ^= 1u;
                }
                ok = ok && bar_wait(barO, parO & 1u, abort);
                if (!ok) {
                    counted = on;
                    break;
                }
                if (on) {
                    const uint32_t M = after(m32), ops = after(ops32), lv = s32(lvl);
                    static_for<0, P>([&](auto nn) {
                        constexpr int n = P - 1 - decltype(nn)::value;
                        constexpr int RT = F::rt(n), KC = F::kc(n), base = n * (n + 1) / 2;
                        const double sc = lds(lv + 8 * n);
                        double v[RT][4] = {};
#pragma unroll
                        for (int kc = 0; kc < KC; ++kc) {
                            const double2 x = lds2(base + 4 * kc + 3 < F::TW ? M + 16 * (base + 4 * kc) : M + 16 * (base + imin(4 * kc + lc, n) - lc));
                            const double fx = e[kc].x * sc, fy = e[kc].y * sc;
                            const double xr = fx * x.x - fy * x.y, xi = fx * x.y + fy * x.x;
#pragma unroll
                            for (int rt = 0; rt < RT; ++rt) {
                                const uint32_t f = ops + (F::rot_off(n) + 2 * (rt * KC + kc)) * 256;
                                dmma(v[rt][0], v[rt][1], lds(f), xr);
                                if (n > 0) dmma(v[rt][2], v[rt][3], lds(f + 256), xi);
                            }
                        }
#pragma unroll
                        for (int rt = 0; rt < RT; ++rt) {
                            if (8 * rt + lr <= n) {
                                unsigned char* o = bufZ + rowm[rt] + 64 * n + st[n & 3];
                                *reinterpret_cast<double2*>(o) = make_double2(v[rt][0], v[rt][1]);
                                *reinterpret_cast<double2*>(o + 64 * F::ZI) = make_double2(v[rt][2], v[rt][3]);
                            }
                        }
                    });
                    ++k;
                    cur = k < na ? act[k] : 255;
                }
                done(0);
                if (on && k < na) {                         // the moments are used up: the next slot's
                    load_moments(src, bufM, 0, F::TW, CS, 0);
                    src = source(k + 1);
                    load_e();
                }
                // the T and I operators of the previous slot are used up: those of slot i + DB - 1 take their place
                if (i > 0) {
                    const int pt = 1 + (i - 1) % DB, pi = 3 + (i - 1) % DB;
                    ok = reload(1, pt, parE >> pt & 1u, i + DB - 1, F::NR, F::NT, S::ops_t + (pt - 1) * 256 * F::NT) &&
                         reload(2, pi, parE >> pi & 1u, i + DB - 1, F::NR + F::NT, F::NI, S::ops_i + (pi - 3) * 256 * F::NI);
                    parE ^= 1u << pt | 1u << pi;
                }
                // ---- T: Lz^k = T_k W^k (in place)
                ok = ok && bar_wait(barO + tb, parO >> tb & 1u, abort);
                if (!ok) break;
                if (on) {
                    const uint32_t z = after(z32 + lc * 64), ops = after(ops32 + (S::ops_t - S::ops) + (tb - 1) * 256 * F::NT);
                    static_for<0, P>([&](auto kk) {
                        constexpr int k = decltype(kk)::value;
                        constexpr int RT = F::trt(k), KC = F::tkc(k), base = F::az(k);
                        double v[RT][4] = {};
#pragma unroll
                        for (int kc = 0; kc < KC; ++kc) {
                            const uint32_t b = z + 64 * (base + 4 * kc) + ld[base & 3];
                            const double br = lds(b), bi = k > 0 ? lds(b + 64 * F::ZI) : 0.0;
#pragma unroll
                            for (int rt = 0; rt < RT; ++rt) {
                                const double f = lds(ops + (F::tz_off(k) + rt * KC + kc) * 256);
                                dmma(v[rt][0], v[rt][1], f, br);
                                if (k > 0) dmma(v[rt][2], v[rt][3], f, bi);
                            }
                        }
#pragma unroll
                        for (int rt = 0; rt < RT; ++rt)
                            if (k + 8 * rt + lr <= P + 1) {
                                unsigned char* o = bufZ + 64 * (base + 8 * rt + lr) + st[base & 3];
                                *reinterpret_cast<double2*>(o) = make_double2(v[rt][0], v[rt][1]);
                                if (k > 0) *reinterpret_cast<double2*>(o + 64 * F::ZI) = make_double2(v[rt][2], v[rt][3]);
                            }
                    });
                }
                done(tb);
                ok = reload(0, 0, parO & 1u, i + 1, 0, F::NR, S::ops);
                // ---- I: S_j += e^{-i m phi} (PB_j Re Lz_j, QB_j Im Lz_j)
                ok = ok && bar_wait(barO + ib, parO >> ib & 1u, abort);
                if (!ok) break;
                if (on) {
                    const uint32_t z = after(z32), ops = after(ops32 + (S::ops_i - S::ops) + (ib - 3) * 256 * F::NI);
                    static_for<0, P + 2>([&](auto jj) {
                        constexpr int j = P + 1 - decltype(jj)::value;
                        constexpr int RT = F::rt(j), KP = F::ikp(j), KQ = F::ikq(j);
                        double v[RT][4] = {};
#pragma unroll
                        for (int kc = 0; kc < KP; ++kc) {
                            const double b = lds(z + rowk[kc] + 64 * j + ld[j & 3]);
#pragma unroll
                            for (int rt = 0; rt < RT; ++rt) dmma(v[rt][0], v[rt][1], lds(ops + (F::inv_off(j) + rt * (KP + KQ) + kc) * 256), b);
                        }
#pragma unroll
                        for (int kc = 0; kc < KQ; ++kc) {
                            const double b = lds(z + rowq[kc] + 64 * (j + F::ZI) + ld[(j + 1) & 3]);
#pragma unroll
                            for (int rt = 0; rt < RT; ++rt)
                                dmma(v[rt][2], v[rt][3], lds(ops + (F::inv_off(j) + rt * (KP + KQ) + KP + kc) * 256), b);
                        }
#pragma unroll
                        for (int rt = 0; rt < RT; ++rt) {
                            double(&u)[4] = sum[F::inv_tiles(j) + rt];
                            const double2 f = c[rt];
                            u[0] += f.x * v[rt][0] + f.y * v[rt][2];
                            u[1] += f.x * v[rt][1] + f.y * v[rt][3];
                            u[2] += f.x * v[rt][2] - f.y * v[rt][0];
                            u[3] += f.x * v[rt][3] - f.y * v[rt][1];
                        }
                    });
#pragma unroll
                    for (int u = 0; u < F::IT; ++u) before(sum[u]);
                }
                done(ib);
                if (on && (k == na || (cur >> 8) / kPartSlots != here)) flush(here);   // the part's last slot
                parO ^= 1u | 1u << tb | 1u << ib;
            }
            if (!ok) {
                parM ^= in_flight(k + counted, imin(k + 1, na), 1);
                *abort = 1;
            }
            if (fresh) flush(part0);                        // no source at all: zeros
        }
        __syncthreads();
        // ================ the order-P sources' part of the potential local
        if (a.want_pot && !*abort) {
            double sum[F::DT][4], v[F::DT][4];              // the sums, and those of the current azimuth
            int azimuth[F::DT], order[F::DT];               // m and order of the lane's row of each tile
#pragma unroll
            for (int u = 0; u < F::DT; ++u) {
                tri_nm(imin(8 * u + lr, T - 1), order[u], azimuth[u]);
#pragma unroll
                for (int h = 0; h < 4; ++h) sum[u][h] = v[u][h] = 0.0;
            }
            constexpr int first = F::NR + F::NT + F::NI;
            auto flush = [&](int part) {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int64_t row = col_row[h], pr = part * g.rows + row - g.node0 * qd;
                    if (row < 0) continue;
                    cplx* out = g.split ? g.part_d + pr * T : a.LA + row * T;
                    cplx old[F::DT];
#pragma unroll
                    for (int t = 0; t < F::DT; ++t) old[t] = !g.split && 8 * t + lr < T ? out[8 * t + lr] : cplx{0, 0};
#pragma unroll
                    for (int t = 0; t < F::DT; ++t) {
                        const double sc = fsc[order[t] + 1];
                        if (8 * t + lr < T) out[8 * t + lr] = cplx{fma(sum[t][h], sc, old[t].re), fma(sum[t][2 + h], sc, old[t].im)};
                    }
                }
#pragma unroll
                for (int t = 0; t < F::DT; ++t) sum[t][0] = sum[t][1] = sum[t][2] = sum[t][3] = 0.0;
            };
            unsigned char* ring = sm + warp * kRing * S::ring_m;
            const uint32_t ring32 = s32(ring) + 16 * (lr * CD);
            proxy_fence();                                   // the stages wrote this space through the generic proxy
            // moments kRing slots ahead, their sources one more
            for (int u = 0; u < kRing; ++u)
                if (u < na) load_moments(source(u), ring + u * S::ring_m, F::TW, P + 1, CD, u);
            int src = source(kRing);
            if (tid == 0)
                for (int u = 0; u < kRing && u < ns; ++u) load_ops(u, first, F::ND, S::ops_d + u * 256 * F::ND, u);
            double2 e[F::DK];                               // s^P e^{i m phi} of the azimuth, m = 4 kc + lc
            uint32_t parE = parO;                           // parities of the operators' earlier uses
            int k = 0, az = -1;
            bool counted = false;                           // as in the first pass
            auto load_e = [&](int s) {
                const double2* eil = phases(s);
#pragma unroll
                for (int kc = 0; kc < F::DK; ++kc) {
                    const double2 f = __ldg(eil + imin(4 * kc + lc, P));
                    e[kc] = make_double2(f.x * lvl[P], f.y * lvl[P]);
                }
            };
            for (int i = 0; i < ns; ++i) {
                const int b = i % kRing, mb = k % kRing;
                const bool on = k < na && (act[k] & 255) == i;
                if (on) {
                    const int s = act[k] >> 8;
                    if (s / 6 != az) load_e(s);
                    az = s / 6;
                    ok = ok && bar_wait(barM + mb, parM >> mb & 1u, abort);
                    parM ^= 1u << mb;
                }
                ok = ok && bar_wait(barO + b, parO >> b & 1u, abort);
                if (!ok) {
                    counted = on;
                    break;
                }
                if (on) {
                    const uint32_t M = after(ring32 + mb * S::ring_m), ops = after(s32(sm + S::ops_d) + lane * 8 + b * 256 * F::ND);
                    double xr[F::DK], xi[F::DK];
#pragma unroll
                    for (int kc = 0; kc < F::DK; ++kc) {
                        const double2 x = lds2(M + 16 * imin(4 * kc + lc, P));
                        xr[kc] = e[kc].x * x.x - e[kc].y * x.y;
                        xi[kc] = e[kc].x * x.y + e[kc].y * x.x;
                    }
                    static_for<0, F::DT>([&](auto tt) {
                        constexpr int t = decltype(tt)::value;
#pragma unroll
                        for (int kc = 0; kc < F::DK; ++kc) {
                            dmma(v[t][0], v[t][1], lds(ops + 2 * (t * F::DK + kc) * 256), xr[kc]);
                            dmma(v[t][2], v[t][3], lds(ops + (2 * (t * F::DK + kc) + 1) * 256), xi[kc]);
                        }
                    });
#pragma unroll
                    for (int u = 0; u < F::DT; ++u) before(v[u]);
                    ++k;
                    if (k == na || (act[k] >> 8) / 6 != az) {    // the azimuth's last slot
                        const double2* eil = phases(act[k - 1] >> 8);
#pragma unroll
                        for (int t = 0; t < F::DT; ++t) {
                            const double2 f = __ldg(eil + azimuth[t]);
                            sum[t][0] += f.x * v[t][0] + f.y * v[t][2];
                            sum[t][1] += f.x * v[t][1] + f.y * v[t][3];
                            sum[t][2] += f.x * v[t][2] - f.y * v[t][0];
                            sum[t][3] += f.x * v[t][3] - f.y * v[t][1];
                            v[t][0] = v[t][1] = v[t][2] = v[t][3] = 0.0;
                        }
                        const int here = (act[k - 1] >> 8) / kPartSlots;
                        if (k == na || (act[k] >> 8) / kPartSlots != here) flush(here);   // and the part's
                    }
                    // the moments are used up: those kRing slots later take their place
                    __syncwarp();
                    if (k + kRing - 1 < na) load_moments(src, ring + mb * S::ring_m, F::TW, P + 1, CD, mb);
                    src = source(k + kRing);
                }
                done(b);
                parO ^= 1u << b;
                // the operators of slot i - 1 are used up: slot i + kRing - 1 takes their place
                if (i > 0) {
                    const int pb = (i - 1) % kRing;
                    ok = reload(i % NW, pb, parE >> pb & 1u, i + kRing - 1, first, F::ND, S::ops_d + pb * 256 * F::ND);
                    parE ^= 1u << pb;
                }
            }
            if (!ok) {
                parM ^= in_flight(k + counted, imin(k + kRing, na), kRing);
                *abort = 1;
            }
            if (g.split && na == 0) flush(part0);
        }
        __syncthreads();
        if (*abort) {
            // copies in flight land before shared memory is released; an operator buffer's copies come from several warps
            if (lane == 0) drain_copies(parM, kRing, kDrainPolls, [&](int b, uint32_t parity) { return bar_try(barM + b, parity); });
            if (tid == 0) {
                atomicExch(a.wait_err, 1);
                *ns_s = 0;
            }
            __syncthreads();
            if (lane == 0) atomicXor(ns_s, static_cast<int>(parO >> kIssued));
            __syncthreads();
            if (tid == 0)
                drain_copies(static_cast<uint32_t>(*ns_s), kOps, kDrainPolls, [&](int b, uint32_t parity) { return bar_try(barO + b, parity); });
            break;
        }
    }
}

template<int P, int NW>
bool launch_w(const EvalArgs& a, const TileArgs& g, int sms, cudaStream_t st)
{
    constexpr size_t smem = Smem<P, NW>::total;
    static_assert(smem <= 227 * 1024, "the tile's working set exceeds shared memory");
    allow_max_smem(k_m2l_tile<P, NW>);
    int per_sm = 0;
    SFMM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_m2l_tile<P, NW>, 32 * NW, smem));
    if (per_sm < 1) return false;
    per_sm = std::min(per_sm, max_per_sm(NW));
    const unsigned grid = static_cast<unsigned>(std::max<int64_t>(1, std::min<int64_t>(g.items, int64_t(sms) * per_sm)));
    SFMM_CUDA(cudaMemsetAsync(g.ctr, 0, sizeof(int), st));
    k_m2l_tile<P, NW><<<grid, 32 * NW, smem, st>>>(a, g);
    SFMM_CHECK_LAUNCH();
    return true;
}

template<int P>
bool launch_p(const EvalArgs& a, const TileArgs& g, int warps, int sms, cudaStream_t st)
{
    if constexpr (P <= kNarrowMaxOrder)
        if (warps == kSmallWarps) return launch_w<P, kSmallWarps>(a, g, sms, st);
    return launch_w<P, full_warps(P)>(a, g, sms, st);
}

}  // namespace tile
}  // namespace sfmm
