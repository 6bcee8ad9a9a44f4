// Host check of offset_class (pd_gpu1_gb300/csrc/bondtpl.h) against
// offset_pair: on random float vectors over the binades 2^-74 to 2^97 and
// doubles near them (steps of 0 to 2^50 ulps, the neighbouring binades, the
// other sign, zero, infinities, NaN), whatever offset_class takes has to be
// offset_pair's pair bit for bit, and it has to take every offset below 2^48
// ulps within the binade.
#include <cmath>
#include <cstdio>
#include <random>

#include "bondtpl.h"

using namespace pdg::bt;

int main() {
    std::mt19937_64 rng(11);
    long bad = 0, taken = 0;
    auto check = [&](double d, float xf) {
        const uint64_t xb = dbits((double)xf);
        f2 got, want;
        const bool ok = offset_class(d, xb, class_scale(xf), got);
        const int64_t df = (int64_t)(dbits(d) - xb);
        const bool usual = ((dbits(d) ^ xb) >> 52) == 0 && df < (1ll << 48) && df >= -(1ll << 48);
        bool fine = ok == usual;
        if (ok) {
            taken++;
            fine = fine && offset_pair(d, xb, want) && fbits(got.h) == fbits(want.h) && fbits(got.l) == fbits(want.l);
        }
        if (!fine && bad++ < 10) printf("d %a xf %a: taken %d, usual %d\n", d, (double)xf, ok, usual);
    };
    for (long k = 0; k < 4000000; k++) {
        const uint32_t m = (uint32_t)rng();
        const float xf = ffrom((m & 0x807fffffu) | (uint32_t)((127 - 74 + rng() % 172) << 23));
        const int64_t step = (int64_t)(rng() >> (13 + rng() % 51));
        const uint64_t xb = dbits((double)xf);
        check(dfrom(k & 1 ? xb + (uint64_t)step : xb - (uint64_t)step), xf);
        if (k % 16 == 0) {
            check((double)xf, xf);
            check(-(double)xf, xf);
            check(2.0 * xf, xf);
            check(0.0, xf);
            check(INFINITY, xf);
            check(NAN, xf);
        }
    }
    printf("%ld offsets taken, %ld differ\n", taken, bad);
    return bad || taken < 1000000 || class_scale(0.0f) != 0.0f || class_scale(1e-30f) != 0.0f;
}
