// Host check of the stretch of the 3-D bond kernels and the state-based passes
// (pd_gpu1_gb300/csrc/bondtpl.h: squares, extension, stretch_ratio, rsqrt2,
// exceeds_near) on bond vectors from D = fl(P_c - P_i) and the positions'
// rounding errors, against quadruple precision.
//
// Bonds of 2-D and 3-D lattices (coordinates (i + 1/2) dx - L/2, horizon 3.015
// dx) under strains from 1e-7 to 3e-2, with and without a rotation that leaves
// the vectors outside their classes' binades.  Bounds, relative to the strain
// scale strain l0 (or the extension where larger): 2e-13 for the pair arithmetic
// (the bound of bondtpl_check) plus the rounding of D, sqrt(N) 2^-53 / strain
// (|D| is at most l0 or so), and, where only the row's own rounding error enters
// (the force of the 3-D bonds, whose neighbour's P the reference rounds too),
// sqrt(N) 2^-53 |P| / (strain l0).
// Where the fast sums may be used they give the general ones' bits.
#include <quadmath.h>

#include <array>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>

#include "bondtpl.h"

using namespace pdg::bt;
typedef __float128 q;

static q qabs(q v) { return v < 0 ? -v : v; }

template <int N, class TT>
static void make(TT& T, const double* xa, double l0t) {
    q s = 0;
    for (int a = 0; a < N; a++) {
        T.xf[a] = (float)xa[a];
        T.xd[a] = dbits((double)T.xf[a]);
        T.sc[a] = class_scale(T.xf[a]);
        s += (q)T.xf[a] * (q)T.xf[a];
    }
    const q c = s - (q)l0t * (q)l0t;
    f2 sp = split_bits((double)s), cp = split_bits((double)c);
    sp.l = (float)((q)sp.l + (s - (q)(double)s));
    cp.l = (float)((q)cp.l + (c - (q)(double)c));
    T.q0h = sp.h, T.q0l = sp.l, T.c0h = cp.h, T.c0l = cp.l;
    const f2 lp = split_bits(l0t);
    T.l0h = lp.h, T.l0l = lp.l, T.l0d = l0t;
}

// x + u - P by the larger of the two, as the kernels keep it.
static float residual(double x, double u, double P) {
    const bool small = std::fabs(x) < std::fabs(u);
    const double hi = small ? u : x, lo = small ? x : u;
    return (float)((hi - P) + lo);
}

static long bits_checked = 0, bits_differ = 0, decisions = 0, wrong = 0;
static double worst = 0.0;  // error over its bound

static void judge(q err, double bound) {
    const double r = (double)err / bound;
    if (!(r <= worst)) worst = r;
}

template <int N, class TT>
static void lattice(double dx, double strain, double rot, std::mt19937_64& rng) {
    std::uniform_real_distribution<double> U(-1.0, 1.0);
    const int n = N == 2 ? 500 : 90, rows = 500;
    const double L = n * dx, delta = 3.015 * dx;
    auto coord = [&](int i) { return (i + 0.5) * dx - L / 2; };
    std::vector<std::array<int, 3>> offs;
    const int zr = N == 3 ? 3 : 0;
    for (int oz = -zr; oz <= zr; oz++)
        for (int oy = -3; oy <= 3; oy++)
            for (int ox = -3; ox <= 3; ox++)
                if ((ox || oy || oz) && dx * dx * (ox * ox + oy * oy + oz * oz) < delta * delta)
                    offs.push_back({ox, oy, oz});
    std::vector<std::array<int, 3>> R(rows);
    for (auto& v : R)
        for (int a = 0; a < 3; a++) v[a] = 3 + (int)(rng() % (n - 6));
    auto reference = [&](int k, size_t o, double* xa) {
        double l2 = 0.0;
        for (int a = 0; a < N; a++) xa[a] = coord(R[k][a] + offs[o][a]) - coord(R[k][a]), l2 += xa[a] * xa[a];
        return std::sqrt(l2);
    };
    std::vector<TT> cls(offs.size());
    for (size_t o = 0; o < offs.size(); o++) {
        double least = 1e300, first[3], xa[3];
        for (int k = 0; k < rows; k++) {
            least = std::min(least, reference(k, o, xa));
            if (k == 0) memcpy(first, xa, sizeof(first));
        }
        make<N>(cls[o], first, least);
    }
    for (int k = 0; k < rows; k++) {
        double g[3][3];
        for (auto& r : g)
            for (auto& v : r) v = strain * U(rng);
        g[0][1] -= rot, g[1][0] += rot;
        for (size_t o = 0; o < offs.size(); o++) {
            const TT& T = cls[o];
            double xa[3], D[3];
            float rc[3], ri[3];
            const double l0 = reference(k, o, xa), dlv = l0 - T.l0d;
            const float dl = (float)dlv;
            if ((double)dl != dlv) continue;
            q dv[3], l2 = 0;
            double pmax = 0.0;
            for (int a = 0; a < N; a++) {
                const double xi = coord(R[k][a]), xc = coord(R[k][a] + offs[o][a]);
                double ui = 0.1 * strain * dx * U(rng), uc = 0.1 * strain * dx * U(rng);
                for (int b = 0; b < N; b++) {
                    ui += g[a][b] * coord(R[k][b]);
                    uc += g[a][b] * coord(R[k][b] + offs[o][b]);
                }
                const double pi = xi + ui, pc = xc + uc;
                D[a] = pc - pi;
                rc[a] = residual(xc, uc, pc), ri[a] = residual(xi, ui, pi);
                pmax = std::fmax(pmax, std::fabs(pc));
                dv[a] = (q)xc + (q)uc - (q)xi - (q)ui;
                l2 += dv[a] * dv[a];
            }
            const q Lq = sqrtq(l2), eq = Lq - (q)l0;
            const q scale = qabs(eq) > (q)(strain * l0) ? qabs(eq) : (q)(strain * l0);
            for (int both = 0; both < 2; both++) {
                f2 eta[3], w[3], d, L2;
                bool ordered = true;
                for (int a = 0; a < N; a++) {
                    if (T.sc[a] == 0.0f)
                        eta[a] = split_bits(D[a]);
                    else if (!offset_class(D[a], T.xd[a], T.sc[a], eta[a]))
                        ordered = false;
                }
                if (!ordered)
                    for (int a = 0; a < N; a++)
                        if (T.xd[a] == 0)
                            eta[a] = split_bits(D[a]);
                        else if (!offset_pair(D[a], T.xd[a], eta[a]))
                            eta[a] = split_bits(D[a] - dfrom(T.xd[a]));
                for (int a = 0; a < N; a++) eta[a].l += both ? rc[a] - ri[a] : -ri[a];
                squares<N, false>(eta, T, dl, w, d, L2);
                if (ordered) {
                    f2 wo[3], dd, LL;
                    squares<N, true>(eta, T, dl, wo, dd, LL);
                    bits_checked++;
                    if (memcmp(wo, w, N * sizeof(f2)) || memcmp(&dd, &d, sizeof(f2)) || memcmp(&LL, &L2, sizeof(f2)))
                        bits_differ++;
                }
                const double bound = 2e-13 + std::sqrt((double)N) * std::ldexp(1.0, -53) *
                                                 (2.0 + (both ? 0.0 : pmax / l0)) / strain;
                const f2 e = extension(d, L2, T, dl), y = rsqrt2(L2);
                judge(qabs((q)e.h + (q)e.l - eq) / scale, bound);
                float eh;
                const f2 g2 = stretch_ratio(d, L2, T, eh), t = mul(e, y);
                q s1 = 0, s2 = 0;  // e d / L by the ratio and by e and 1 / L
                for (int a = 0; a < N; a++) {
                    const q W = (q)w[a].h + (q)w[a].l, want = eq * dv[a] / Lq;
                    const q v1 = ((q)g2.h + (q)g2.l) * W - want, v2 = ((q)t.h + (q)t.l) * W - want;
                    s1 += v1 * v1, s2 += v2 * v2;
                }
                judge(sqrtq(s1) / scale, bound);
                judge(sqrtq(s2) / scale, bound);
                // break decisions at thresholds from far to a unit of the last place away
                const double s = ((double)e.h + (double)e.l) / l0;
                const float eh2 = prod(d.h, rcp_seed(fmaf(L2.h, y.h, T.l0h)));
                for (int b = -53; b <= -1; b += 4) {
                    const double s0 = s * (1.0 + (rng() & 1 ? 1.0 : -1.0) * std::ldexp(1.0, b));
                    if (!(s0 > 0.0)) continue;
                    const bool want = (double)e.h + (double)e.l > s0 * (T.l0d + (double)dl);
                    decisions += 2;
                    wrong += exceeds_near(eh, d, L2, s0, (float)s0, T, dl) != want;
                    wrong += exceeds_near(eh2, d, L2, s0, (float)s0, T, dl) != want;
                }
            }
        }
    }
}

int main() {
    std::mt19937_64 rng(77);
    for (double dx : {5e-5, 1e-3, 0.25})
        for (double strain : {1e-7, 1e-5, 1e-3, 3e-2})
            for (double rot : {0.0, 0.2}) {
                lattice<2, Tpl>(dx, strain, rot, rng);
                lattice<3, Tpl3>(dx, strain, rot, rng);
            }
    std::printf("worst error over its bound: %.3f\n", worst);
    std::printf("fast sums: %ld checked, %ld differ\n", bits_checked, bits_differ);
    std::printf("break decisions: %ld checked, %ld differ\n", decisions, wrong);
    return worst <= 1.0 && bits_checked > 100000 && bits_differ == 0 && decisions > 100000 && wrong == 0 ? 0 : 1;
}
