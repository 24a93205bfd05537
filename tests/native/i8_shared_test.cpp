// CPU checks of the tensor-core M2L's shared rows (simplefmm_b200/csrc/i8_ops.h):
// where they are used, every column has one position, and a coefficient's
// potential and field rows have the same entries for source orders < p and the
// same largest scaled entry (so the same digits).
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <vector>

#include "fmm_tables.h"
#include "i8_ops.h"

using namespace sfmm;

int main()
{
    int fails = 0;
    for (int p = 2; p <= kI8MaxOrder; ++p) {
        const bool shared = i8_shared_rows(p);
        const int RA = (p + 1) * (p + 1), KB = (p * p + 31) / 32, KS = shared ? KB + 1 : (RA + 31) / 32;
        std::vector<int> seen(RA, 0);
        for (int pos = 0; pos < 32 * KS; ++pos) {
            const int k = i8_column(pos, p, KB, shared);
            if (k < 0) continue;
            int n, m, im;
            real_nm(k, n, m, im);
            if (k >= RA || (shared && (n == p) != (pos >= 32 * KB))) ++fails;
            else ++seen[k];
        }
        for (int v : seen) fails += v != 1;
        if (!shared) continue;
        const DirectTables h = make_direct_tables(p);
        const DirectArgs da{h.coef.data(), h.ncoef, h.zil.data(), h.nz, reinterpret_cast<const cplx*>(h.eil2.data()), h.ne};
        for (int r = 0; r < RA; ++r) {
            double ba = 0, bb = 0;
            for (int c = 0; c < 343; ++c) {
                if (!offset_valid(c)) continue;
                for (int k = 0; k < RA; ++k) {
                    int n, m, im;
                    real_nm(k, n, m, im);
                    const double a = op_entry(da, p, RA, c, r, k), b = op_entry(da, p, RA, c, RA + r, k);
                    fails += n < p ? a != b : b != 0.0;
                    ba = std::max(ba, std::fabs(a) * i8_gamma(n));
                    bb = std::max(bb, std::fabs(b) * i8_gamma(n));
                }
            }
            if (ba != bb) {
                std::printf("p %d row %d: %.17g vs %.17g\n", p, r, ba, bb);
                ++fails;
            }
        }
    }
    std::printf(fails ? "i8 shared rows: %d failures\n" : "i8 shared ok\n", fails);
    return fails != 0;
}
