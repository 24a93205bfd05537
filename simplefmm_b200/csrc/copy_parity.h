// Which phase of an mbarrier to wait for so that every bulk copy issued to it
// has landed (host and device; tests/native/copy_parity_test.cpp).
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define SFMM_CP_HD __host__ __device__ __forceinline__
#else
#define SFMM_CP_HD inline
#endif

namespace sfmm {

// `issued`: bit b flips with every copy issued to barrier b, one phase of the
// barrier per copy, so after k copies the last phase is k - 1 and has parity
// bit b ^ 1.  Waiting on that parity returns at once where nothing was ever
// issued (a fresh barrier reports odd phases complete) and where the last copy
// has landed; else when it lands.  The other parity never completes.
SFMM_CP_HD uint32_t last_copy_parity(uint32_t issued, int b) { return (issued >> b & 1u) ^ 1u; }

// The bits of a warp that gives up, from those of its waits: of a pass's copies,
// in turn on `ring` barriers, the first `waited` were waited for (or counted as
// such) and `issued` issued; the rest flip their barrier's bit.
SFMM_CP_HD uint32_t in_flight(int waited, int issued, int ring)
{
    uint32_t bits = 0;
    for (int s = waited; s < issued; ++s) bits ^= 1u << (s % ring);
    return bits;
}

// Waits for barriers 0 .. n - 1 with at most `polls` polls each; try_wait(b,
// parity) is one poll.  False when a barrier's polls ran out.
template<typename TryWait>
SFMM_CP_HD bool drain_copies(uint32_t issued, int n, int polls, TryWait try_wait)
{
    bool ok = true;
    for (int b = 0; b < n; ++b) {
        bool landed = false;
        for (int it = 0; it < polls && !landed; ++it) landed = try_wait(b, last_copy_parity(issued, b));
        ok &= landed;
    }
    return ok;
}

}  // namespace sfmm
