// copy_parity.h against a model of an mbarrier with one arrival a phase:
// random orders of issue, landing and waiting, cut off anywhere.
#include <cstdio>
#include <random>

#include "copy_parity.h"

struct Barrier {
    long issued = 0, landed = 0;          // phases begun (a copy issued), phases complete
    // true iff the phase of that parity before the current one is complete
    bool try_wait(unsigned parity) const { return (landed & 1) != long(parity & 1); }
};

int main()
{
    std::mt19937 rng(7);
    long checked = 0, flying = 0;
    for (int run = 0; run < 20000; ++run) {
        constexpr int n = 5;
        Barrier bar[n];
        unsigned issued = 0;
        const int steps = rng() % 60;
        for (int s = 0; s < steps; ++s) {
            const int b = rng() % n;
            if (bar[b].issued == bar[b].landed) {         // the next copy only after the last one has landed
                issued ^= 1u << b;
                ++bar[b].issued;
            } else if (rng() % 2) {
                ++bar[b].landed;
            }
        }
        // nothing lands any more: exactly the barriers with a copy in flight run out of polls
        int out = 0;
        for (int b = 0; b < n; ++b) {
            int polls = 0;
            sfmm::drain_copies(issued >> b & 1u, 1, 50, [&](int, unsigned p) { ++polls; return bar[b].try_wait(p); });
            out += polls == 50;
            if ((polls == 50) != (bar[b].issued > bar[b].landed) || (polls != 50 && polls != 1)) {
                std::printf("barrier %d: %d polls, issued %ld landed %ld\n", b, polls, bar[b].issued, bar[b].landed);
                return 1;
            }
        }
        // the copies land while the drain polls: it returns true, no earlier than the last landing
        long polls = 0;
        const bool ok = sfmm::drain_copies(issued, n, 50, [&](int b, unsigned p) {
            ++polls;
            if (rng() % 4 == 0 && bar[b].landed < bar[b].issued) ++bar[b].landed;
            return bar[b].try_wait(p);
        });
        for (int b = 0; b < n; ++b)
            if (ok && bar[b].landed != bar[b].issued) return 2;
        if (!ok && polls < 50) return 3;
        if (out == 0 && polls != n) return 4;
        checked += ok;
        flying += out > 0;
    }
    if (checked < 15000 || flying < 5000) return 5;
    // passes of na copies in turn on `ring` barriers, `ring` ahead, given up before or after the wait for copy k: the
    // waits' bits and in_flight give the issues' bits
    for (int ring : {1, 2, 4})
        for (int na = 0; na < 12; ++na)
            for (int stop = 0; stop <= na; ++stop)
                for (int counted = 0; counted <= (stop < na); ++counted) {
                    unsigned waits = rng() & ((1u << ring) - 1), issues = waits;   // bits left by earlier passes: all landed
                    auto issue = [&](int s) { issues ^= 1u << (s % ring); };
                    for (int s = 0; s < ring && s < na; ++s) issue(s);
                    for (int k = 0; k < stop; ++k) {
                        waits ^= 1u << (k % ring);
                        if (k + ring < na) issue(k + ring);
                    }
                    if (counted) waits ^= 1u << (stop % ring);
                    const int issued = stop + ring < na ? stop + ring : na;
                    if ((waits ^ sfmm::in_flight(stop + counted, issued, ring)) != issues) return 6;
                }
    std::printf("copy parity ok\n");
    return 0;
}
