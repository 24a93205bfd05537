// Direct FP64 sums at selected targets -- the reference's accuracy check
// (main.cpp:70-111) on the device: two targets per thread, source records
// staged in shared memory and read by broadcast.  Used to state the FMM error
// against the exact sum.
//
// Bound: the FP64 pipe, about 20 instructions a pair with 1/r from rsqrt and no
// division: 10,000 targets x 400,000 points 6.0 ms (the call 29.2 -> 6.5 ms);
// 28.1 ms with a square root, a division by r and three by r^3 a pair and one
// target per thread.
#include "fmm_internal.cuh"

#include <algorithm>
#include <mutex>

namespace sfmm {

std::atomic<long long> g_launches{0};

namespace {

constexpr int kThreads = 128;
constexpr int kPerThread = 2;                             // targets per thread
constexpr int kTargets = kThreads * kPerThread;           // targets per block
constexpr int kTile = 128;                                // sources per tile

// One staged tile against the thread's targets.  SELF: some target of the warp
// is among the tile's sources; ks is its slot (the pair is left out).
template<int QD, bool SELF>
__device__ __forceinline__ void direct_tile(const double4* __restrict__ s4, const double2* __restrict__ s2, int cnt,
                                            const double (&x)[kPerThread][3], const int64_t (&ks)[kPerThread],
                                            double (&pa)[kPerThread][QD], double (&fa)[kPerThread][3])
{
#pragma unroll 2
    for (int k = 0; k < cnt; ++k) {
        const double4 v = s4[k];
        const double2 w = QD > 1 ? s2[k] : make_double2(0, 0);
#pragma unroll
        for (int u = 0; u < kPerThread; ++u) {
            if (SELF && k == ks[u]) continue;
            const double dx = x[u][0] - v.x, dy = x[u][1] - v.y, dz = x[u][2] - v.z;
            const double ir = rsqrt(fma(dx, dx, fma(dy, dy, dz * dz)));
            const double ir3 = ir * ir * ir;
            pa[u][0] = fma(v.w, ir, pa[u][0]);
            if (QD > 1) pa[u][1] = fma(w.x, ir, pa[u][1]);
            if (QD > 2) pa[u][2] = fma(w.y, ir, pa[u][2]);
            if (QD == 1) {
                const double c = v.w * ir3;
                fa[u][0] = fma(c, dx, fa[u][0]);
                fa[u][1] = fma(c, dy, fa[u][1]);
                fa[u][2] = fma(c, dz, fa[u][2]);
            } else if (QD == 3) {
                fa[u][0] = fma(w.x * dz - w.y * dy, ir3, fa[u][0]);
                fa[u][1] = fma(w.y * dx - v.w * dz, ir3, fa[u][1]);
                fa[u][2] = fma(v.w * dy - w.x * dx, ir3, fa[u][2]);
            }
        }
    }
}

// A target's field again, from the unit vectors R / r: q / r^3 leaves the range
// of the type where q / r^2 does not (pairs closer than 1e-102, say, or charges
// of 1e-150 at 1e60).  Only targets whose potential is finite and whose field is
// not, or whose potential is below 1e-90, come here: q / r^3 below the type's
// normal numbers means q / r below 1e-102 for every r whose cube is in range.
template<int QD>
__device__ __noinline__ void direct_field_in_range(const double* __restrict__ xyz, const double* __restrict__ Q, int64_t jb, int64_t je,
                                                   int64_t i, double (&f)[3])
{
    const double x = xyz[3 * i], y = xyz[3 * i + 1], z = xyz[3 * i + 2];
    f[0] = f[1] = f[2] = 0.0;
    for (int64_t j = jb; j < je; ++j) {
        if (j == i) continue;
        const double dx = x - xyz[3 * j], dy = y - xyz[3 * j + 1], dz = z - xyz[3 * j + 2];
        const double r = sqrt(fma(dx, dx, fma(dy, dy, dz * dz)));
        const double ex = dx / r, ey = dy / r, ez = dz / r;
        const double* q = Q + j * QD;
        if (QD == 1) {
            f[0] += q[0] / r * ex / r;
            f[1] += q[0] / r * ey / r;
            f[2] += q[0] / r * ez / r;
        } else if (QD == 3) {
            f[0] += (q[1] * ez - q[2] * ey) / r / r;
            f[1] += (q[2] * ex - q[0] * ez) / r / r;
            f[2] += (q[0] * ey - q[1] * ex) / r / r;
        }
    }
}

template<int QD>
__global__ void __launch_bounds__(kThreads) k_direct(const double* __restrict__ xyz, int64_t n, const double* __restrict__ Q,
                                                     const int64_t* __restrict__ targets, int64_t nt, int64_t chunk,
                                                     double* __restrict__ part)
{
    __shared__ double4 s4[kTile];
    __shared__ double2 s2[QD > 1 ? kTile : 1];
    int64_t t[kPerThread], i[kPerThread];
    bool on[kPerThread];
    double x[kPerThread][3], pa[kPerThread][QD] = {}, fa[kPerThread][3] = {};
#pragma unroll
    for (int u = 0; u < kPerThread; ++u) {
        t[u] = blockIdx.x * int64_t(kTargets) + u * kThreads + threadIdx.x;
        const int64_t ti = t[u] < nt ? targets[t[u]] : -1;
        // a target index outside [0, n) reads nothing; k_direct_sum reports it
        on[u] = ti >= 0 && ti < n;
        i[u] = on[u] ? ti : -1;
#pragma unroll
        for (int c = 0; c < 3; ++c) x[u][c] = on[u] ? xyz[3 * i[u] + c] : 0.0;
    }
    // sources [jb, je) of this block's chunk (blockIdx.y)
    const int64_t jb = blockIdx.y * chunk;
    const int64_t je = jb + chunk < n ? jb + chunk : n;
    for (int64_t j0 = jb; j0 < je; j0 += kTile) {
        const int cnt = je - j0 < kTile ? static_cast<int>(je - j0) : kTile;
        __syncthreads();
        for (int k = threadIdx.x; k < cnt; k += kThreads) {
            const int64_t j = j0 + k;
            s4[k] = make_double4(xyz[3 * j], xyz[3 * j + 1], xyz[3 * j + 2], Q[j * QD]);
            if (QD > 1) s2[k] = make_double2(Q[j * QD + 1], QD > 2 ? Q[j * QD + QD - 1] : 0.0);
        }
        __syncthreads();
        int64_t ks[kPerThread];
        bool self = false;
#pragma unroll
        for (int u = 0; u < kPerThread; ++u) {
            ks[u] = i[u] - j0;
            self |= ks[u] >= 0 && ks[u] < cnt;
        }
        if (__any_sync(0xffffffffu, self))
            direct_tile<QD, true>(s4, s2, cnt, x, ks, pa, fa);
        else
            direct_tile<QD, false>(s4, s2, cnt, x, ks, pa, fa);
    }
#pragma unroll
    for (int u = 0; u < kPerThread; ++u) {
        if (!on[u]) continue;
        double ps = 0.0;
#pragma unroll
        for (int b = 0; b < QD; ++b) ps += fabs(pa[u][b]);
        const bool in_range = isfinite(fa[u][0]) && isfinite(fa[u][1]) && isfinite(fa[u][2]);
        if (QD != 2 && isfinite(ps) && (!in_range || (ps > 0.0 && ps < 1e-90)))
            direct_field_in_range<QD>(xyz, Q, jb, je, i[u], fa[u]);
        double* o = part + (blockIdx.y * nt + t[u]) * 6;
        for (int b = 0; b < 3; ++b) o[b] = b < QD ? pa[u][b < QD ? b : 0] : 0.0;
        for (int c = 0; c < 3; ++c) o[3 + c] = fa[u][c];
    }
}

// Source chunks: enough blocks to fill the device several times over, at least
// 512 sources each, at most `most` chunks.
int64_t direct_chunks(int64_t n, int64_t nt, int sms, int64_t most)
{
    const int64_t gx = (nt + kTargets - 1) / kTargets;
    const int64_t want = std::max<int64_t>(1, (int64_t(sms) * 16 + gx - 1) / gx);
    return std::max<int64_t>(1, std::min(std::min(want, std::max<int64_t>(1, n / 512)), std::min<int64_t>(most, 65535)));
}

void launch_direct(const double* xyz, int64_t n, const double* Q, int qdim, const int64_t* targets, int64_t nt, int64_t nchunk,
                   double* part, cudaStream_t st)
{
    const int64_t chunk = (n + nchunk - 1) / nchunk;
    const dim3 grid(static_cast<unsigned>((nt + kTargets - 1) / kTargets), static_cast<unsigned>(nchunk));
    if (qdim == 1) k_direct<1><<<grid, kThreads, 0, st>>>(xyz, n, Q, targets, nt, chunk, part);
    else if (qdim == 2) k_direct<2><<<grid, kThreads, 0, st>>>(xyz, n, Q, targets, nt, chunk, part);
    else k_direct<3><<<grid, kThreads, 0, st>>>(xyz, n, Q, targets, nt, chunk, part);
    SFMM_CHECK_LAUNCH();
}

// Sum the chunks' partial sums in chunk order (deterministic).  A target
// index outside [0, n) gets NaN outputs and sets *bad (when given).
__global__ void k_direct_sum(const double* __restrict__ part, int64_t nt, int nchunk, int qdim,
                             const int64_t* __restrict__ targets, int64_t n, double* __restrict__ pot,
                             double* __restrict__ field, int* __restrict__ bad)
{
    const int64_t t = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (t >= nt) return;
    const int64_t ti = targets[t];
    if (ti < 0 || ti >= n) {
        const double nan = __longlong_as_double(0x7ff8000000000000LL);
        if (pot)
            for (int b = 0; b < qdim; ++b) pot[t * qdim + b] = nan;
        if (field)
            for (int c = 0; c < 3; ++c) field[t * 3 + c] = nan;
        if (bad) atomicOr(bad, 1);
        return;
    }
    double acc[6] = {0, 0, 0, 0, 0, 0};
    for (int c = 0; c < nchunk; ++c)
        for (int k = 0; k < 6; ++k) acc[k] += part[(c * nt + t) * 6 + k];
    if (pot)
        for (int b = 0; b < qdim; ++b) pot[t * qdim + b] = acc[b];
    if (field)
        for (int c = 0; c < 3; ++c) field[t * 3 + c] = acc[3 + c];
}

}  // namespace

void direct_sum(Context& c, const double* xyz, int64_t n, const double* Q, int qdim, const int64_t* targets, int64_t nt,
                double* pot, double* field, int* bad)
{
    if (nt <= 0) return;
    const int64_t nchunk = direct_chunks(n, nt, c.sm_count, 65535);
    DevBuf<double> part;
    part.alloc(size_t(nchunk) * nt * 6, c.stream);
    launch_direct(xyz, n, Q, qdim, targets, nt, nchunk, part.ptr, c.stream);
    k_direct_sum<<<static_cast<unsigned>((nt + 255) / 256), 256, 0, c.stream>>>(
        part.ptr, nt, static_cast<int>(nchunk), qdim, targets, n, pot, field, bad);
    SFMM_CHECK_LAUNCH();
}

}  // namespace sfmm

// ------------------------------------------------------------------ direct sum without allocation
// fmm_direct_noalloc: the same two kernels with their partial sums in a
// fixed, file-scope device array instead of memory allocated per call.  It is
// for callers that cannot allocate device memory while they run: callers that
// hold a fixed device-memory budget for their own lifetime (a solver service
// that admits work against a budget), and callers that cannot wait on an
// allocation (growing a memory pool can stall a call for a long time).
namespace sfmm {
namespace {

// Partial sums: 6 doubles per (source chunk, target).  8 MiB on every device
// that loads this library, held until the process exits.
constexpr int64_t kNoAllocScratchDoubles = int64_t(1) << 20;
constexpr int64_t kNoAllocMaxTargets = kNoAllocScratchDoubles / 6;    // 174,762
static __device__ __align__(256) double g_noalloc_scratch[kNoAllocScratchDoubles];

struct NoAllocDevice {
    double* scratch = nullptr;     // device address of g_noalloc_scratch
    int sms = 0;
};

// Set-up, once per device, with that device current: the device address of
// the scratch array (its host-side name is only a stand-in) and the SM count.
NoAllocDevice noalloc_device(int dev)
{
    static std::mutex mu;
    static NoAllocDevice table[64];
    std::lock_guard<std::mutex> lk(mu);
    NoAllocDevice& d = table[dev];
    if (!d.scratch) {
        double* ptr = nullptr;
        SFMM_CUDA(cudaGetSymbolAddress(reinterpret_cast<void**>(&ptr), g_noalloc_scratch));
        int sms = 0;
        SFMM_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        d.sms = sms;
        d.scratch = ptr;
    }
    return d;
}

}  // namespace
}  // namespace sfmm

extern "C" int fmm_direct_noalloc(const double* xyz, int64_t n, const double* Q, int qdim, const int64_t* targets,
                                  int64_t nt, double* pot, double* field, void* stream)
{
    using namespace sfmm;
    try {
        if (!xyz || !Q || !targets) return record_failure(FMM_ERR_INVALID_ARGUMENT, "NULL argument");
        if (qdim < 1 || qdim > 3) return record_failure(FMM_ERR_UNSUPPORTED, "qdim must be 1, 2 or 3");
        if (field && qdim == 2) return record_failure(FMM_ERR_UNSUPPORTED, "the field needs qdim 1 or 3");
        if (n <= 0 || nt < 0) return record_failure(FMM_ERR_INVALID_ARGUMENT, "bad sizes");
        if (nt > kNoAllocMaxTargets)
            return record_failure(FMM_ERR_OVER_BUDGET,
                                  "fmm_direct_noalloc takes at most 174762 targets per call (8 MiB of fixed scratch)");
        if (nt == 0) return FMM_OK;
        int dev = 0;
        SFMM_CUDA(cudaGetDevice(&dev));
        if (dev < 0 || dev >= 64) return record_failure(FMM_ERR_UNSUPPORTED, "device index above 63");
        const NoAllocDevice d = noalloc_device(dev);
        cudaStream_t st = static_cast<cudaStream_t>(stream);
        // chunking as direct_sum, capped by the scratch size
        const int64_t nchunk = direct_chunks(n, nt, d.sms, kNoAllocScratchDoubles / (6 * nt));
        // every (chunk, target) slot of the scratch is written before it is
        // read, so nothing left by an earlier call needs clearing
        launch_direct(xyz, n, Q, qdim, targets, nt, nchunk, d.scratch, st);
        // a target index outside [0, n) is not read: its outputs become NaN
        k_direct_sum<<<static_cast<unsigned>((nt + 255) / 256), 256, 0, st>>>(
            d.scratch, nt, static_cast<int>(nchunk), qdim, targets, n, pot, field, nullptr);
        SFMM_CHECK_LAUNCH();
        return FMM_OK;
    } catch (const sfmm::Error& e) {
        return record_failure(e.status, e.what());
    } catch (const std::exception& e) {
        return record_failure(FMM_ERR_CUDA, e.what());
    }
}
