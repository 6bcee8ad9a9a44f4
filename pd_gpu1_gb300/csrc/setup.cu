// Setup passes over the CSR bond family, and the build of the SELL-32 layout
// the force kernels read.
//
//   vol_corr          kernel_vol_Corr (Surf_Corr.cu:7-35)
//   surface_correct   surface_correct_gpu (Surf_Corr.cu:235-310): the reference
//                     runs 5-8 launches with a displacement array per test
//                     field and cudaMalloc/cudaFree temporaries; here one
//                     thread per node computes idist, fac and the strain energy
//                     of all test fields at once (u_axis = 0.001 x_axis is
//                     analytic), in a state-based context w and m as well, then
//                     one pass forms scr per bond.
//   initial_weight    kernel_initial_weight_2D/3D (Force_State.cu:8-54), in the
//                     same family pass as vol_corr (k_family_setup)
//   set_crack_*       kernel_set_crack_2D (Base_Function.cu:39-81) and the
//                     Kalthoff-Winkler notch cut (Solve_Kalthoff_Winkler.cu:40-63)
//   prepare           per-bond coefficients in SELL order (see pd_internal.cuh)
//
// This file is compiled without FMA contraction: idist, fac, w and the crack
// tests then round exactly like the reference's host code, so NL, idist, fac
// and the fail flags agree bit for bit with it.
#include <cmath>

#include "ff.cuh"
#include <algorithm>
#include <cmath>

#include "pd_internal.cuh"

namespace pdg {
namespace {

// The order of a warp's shuffle-tree sum over 32 lanes, kept by a single thread:
// leaf j = 0, 16, 8, 24, 4, ... (bit-reversed) and every pair added as soon as
// it is complete gives v_j + v_(j+16), then + 8, 4, 2 and 1.  Four leaves come
// at a time; s[] holds the three upper levels.
struct TreeSum {
    double s[3];
    // the sum of the group's four leaves; true when the tree is complete (v: its sum)
    __device__ __forceinline__ void add(int group, double& v) {
        if (group & 1) {
            v = s[0] + v;
            if (group & 2) {
                v = s[1] + v;
                if (group & 4)
                    v = s[2] + v;
                else
                    s[2] = v;
            } else {
                s[1] = v;
            }
        } else {
            s[0] = v;
        }
    }
};

// One pass over node i's bonds:
//   * idist and fac per bond (kernel_vol_Corr, Surf_Corr.cu:17-32);
//   * with ENERGY, the strain energy density of node i under the test fields
//     u_a = 0.001 x_a (kernel_Disp + kernel_surface_F/_3D, Surf_Corr.cu:38-158),
//     all axes at once, and fncst_a = sedload / energy.  A batch of specimens
//     passes bc and sedload per node (its specimen's values); bonds never
//     cross specimens;
//   * with WEIGHT, w per bond and m per node (kernel_initial_weight_2D/3D,
//     Force_State.cu:8-54).
// The reference runs these as separate passes that re-read idist and fac;
// here they come from registers.  FamilyRow is one row and what its bonds add:
// DIM energy sums, then the weight sum.
template <int DIM, bool ENERGY, bool WEIGHT>
struct FamilyRow {
    static constexpr int NS = ENERGY ? DIM : 0;
    static constexpr int NA = NS + (WEIGHT ? 1 : 0) + (ENERGY || WEIGHT ? 0 : 1);
    double xi[3], ui[3], inner, outer, quarter;

    __device__ __forceinline__ FamilyRow(const KParams& P, const double* __restrict__ x, const double* __restrict__ y,
                                         const double* __restrict__ z, int64_t i)
        : xi{x[i], y[i], DIM == 3 ? z[i] : 0.0},
          ui{0.001 * xi[0], 0.001 * xi[1], 0.001 * xi[2]},
          inner(P.delta - P.dx / 2.0),
          outer(P.delta + P.dx / 2.0),
          quarter(0.25 * P.bc) {}

    // the bond at place q of the CSR arrays, its terms added to leaf
    __device__ __forceinline__ void bond(const KParams& P, const double* __restrict__ x, const double* __restrict__ y,
                                         const double* __restrict__ z, const int* __restrict__ NL, int64_t q,
                                         double* __restrict__ idist, double* __restrict__ fac, double* __restrict__ w,
                                         double (&leaf)[NA]) const {
        const int64_t c = NL[q];
        double xc[3], d[3], sq[3];
#pragma unroll
        for (int a = 0; a < DIM; a++) {
            xc[a] = a == 0 ? x[c] : a == 1 ? y[c] : z[c];
            d[a] = xc[a] - xi[a];
            sq[a] = d[a] * d[a];
        }
        const double L0 = sqrt(DIM == 2 ? sq[0] + sq[1] : sq[0] + sq[1] + sq[2]);
        idist[q] = L0;
        // positive doubles compare like their bit patterns (off the FP64 pipe)
        const long long lb = __double_as_longlong(L0);
        double f;
        if (lb <= __double_as_longlong(inner))
            f = 1.0;
        else if (lb <= __double_as_longlong(outer))
            f = (outer - L0) / P.dx;
        else
            f = 0.0;
        fac[q] = f;
        if (ENERGY) {
#pragma unroll
            for (int a = 0; a < DIM; a++) {
                // displacement only along axis a (the other components are
                // zero, and adding zero is exact, so the reference's expression
                // reduces to the plain coordinate difference on those axes)
                const double dd = xc[a] + 0.001 * xc[a] - xi[a] - ui[a];
                double e[3] = {sq[0], sq[1], DIM == 3 ? sq[2] : 0.0};
                e[a] = dd * dd;
                const double L = sqrt(DIM == 2 ? e[0] + e[1] : e[0] + e[1] + e[2]);
                leaf[a] += quarter * (L - L0) * (L - L0) / L0 * P.vol * f;
            }
        }
        if (WEIGHT) {
            const double wq = exp(-(L0 * L0) / (P.delta * P.delta));
            w[q] = wq;
            leaf[NS] += wq * (L0 * L0) * P.vol * f;
        }
    }

    __device__ __forceinline__ void store(const double (&v)[NA], int64_t i, double sedload, double* __restrict__ fx,
                                          double* __restrict__ fy, double* __restrict__ fz,
                                          double* __restrict__ m) const {
        if (ENERGY) {
            fx[i] = sedload / v[0];
            fy[i] = sedload / v[1];
            if (DIM == 3) fz[i] = sedload / v[NS - 1];
        }
        if (WEIGHT) m[i] = v[NS];
    }
};

// The family pass, one thread per node.  The sums keep the order of a warp per
// node (bonds j, j + 32, ... in lane j, then the shuffle tree), so that the
// results are bit for bit those of k_family_setup_warp; a thread per node issues
// the FP64 additions of the tree for 28 bonds instead of 160 lanes and leaves no
// lanes idle on rows of 28.  Measured on 7.0M 2-D bonds with ENERGY: 2.15 ms with
// a warp per node, 1.16 so; what is left is three square roots and two divisions
// a bond.
template <int DIM, bool ENERGY, bool WEIGHT>
__global__ void __launch_bounds__(128) k_family_setup(KParams P, double sedload, const double* __restrict__ node_bc,
                               const double* __restrict__ node_sed, const double* __restrict__ x,
                               const double* __restrict__ y, const double* __restrict__ z,
                               const int64_t* __restrict__ rowptr, const int* __restrict__ NL,
                               double* __restrict__ idist, double* __restrict__ fac, double* __restrict__ fx,
                               double* __restrict__ fy, double* __restrict__ fz, double* __restrict__ w,
                               double* __restrict__ m) {
    using Row = FamilyRow<DIM, ENERGY, WEIGHT>;
    constexpr int NA = Row::NA;
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= P.N) return;
    if (ENERGY && node_bc) {
        P.bc = node_bc[i];
        sedload = node_sed[i];
    }
    const Row row(P, x, y, z, i);
    const int64_t q0 = rowptr[i];
    const int n = (int)(rowptr[i + 1] - q0);
    TreeSum tree[NA];
    double v[NA];
#pragma unroll 1
    for (int group = 0; group < 8; group++) {
        const int j0 = ((group & 1) << 2) | (group & 2) | (group >> 2);
        double pair[NA], quad[NA];
#pragma unroll 1
        for (int t = 0; t < 4; t++) {  // leaves j0, j0 + 16, j0 + 8, j0 + 24
            double leaf[NA];
#pragma unroll
            for (int a = 0; a < NA; a++) leaf[a] = 0.0;
            for (int j = j0 + ((t & 1) << 4) + ((t & 2) << 2); j < n; j += 32)
                row.bond(P, x, y, z, NL, q0 + j, idist, fac, w, leaf);
            if (ENERGY || WEIGHT) {
#pragma unroll
                for (int a = 0; a < NA; a++) {
                    if (t == 0)
                        pair[a] = leaf[a];
                    else if (t == 1)
                        quad[a] = pair[a] + leaf[a];
                    else if (t == 2)
                        pair[a] = leaf[a];
                    else
                        v[a] = quad[a] + (pair[a] + leaf[a]);
                }
            }
        }
        if (ENERGY || WEIGHT) {
#pragma unroll
            for (int a = 0; a < NA; a++) tree[a].add(group, v[a]);
        }
    }
    row.store(v, i, sedload, fx, fy, fz, m);
}

// The family pass, one warp per node: a small specimen's rows are too few to
// fill the GPU with a thread each, and a thread's bonds come one after the other
// (family_by_warps has where each is the faster one).
template <int DIM, bool ENERGY, bool WEIGHT>
__global__ void __launch_bounds__(256) k_family_setup_warp(KParams P, double sedload, const double* __restrict__ node_bc,
                               const double* __restrict__ node_sed, const double* __restrict__ x,
                               const double* __restrict__ y, const double* __restrict__ z,
                               const int64_t* __restrict__ rowptr, const int* __restrict__ NL,
                               double* __restrict__ idist, double* __restrict__ fac, double* __restrict__ fx,
                               double* __restrict__ fy, double* __restrict__ fz, double* __restrict__ w,
                               double* __restrict__ m) {
    using Row = FamilyRow<DIM, ENERGY, WEIGHT>;
    constexpr int NA = Row::NA;
    const int64_t i = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (i >= P.N) return;
    if (ENERGY && node_bc) {
        P.bc = node_bc[i];
        sedload = node_sed[i];
    }
    const Row row(P, x, y, z, i);
    const int64_t q1 = rowptr[i + 1];
    double v[NA];
#pragma unroll
    for (int a = 0; a < NA; a++) v[a] = 0.0;
    for (int64_t q = rowptr[i] + lane; q < q1; q += 32) row.bond(P, x, y, z, NL, q, idist, fac, w, v);
    if (ENERGY || WEIGHT) {
#pragma unroll
        for (int a = 0; a < NA; a++)
            for (int off = 16; off > 0; off >>= 1) v[a] += __shfl_down_sync(0xffffffffu, v[a], off);
        if (lane == 0) row.store(v, i, sedload, fx, fy, fz, m);
    }
}

// The squared direction cosines of a bond, cos^2 and sin^2 of the reference's
// angle expressions, remembered by the bit patterns of their operands.  On a
// lattice a few thousand operand pairs serve every bond (a coordinate
// difference takes a handful of roundings per offset), and the trigonometric
// functions, several hundred FP64 instructions a bond, were most of the pass.
// A slot's first key word is 0 (empty), kBusy while its values are written, or
// the key; whoever finds no slot ready computes the values itself.
struct TrigSlot {
    unsigned long long ka, kb;
    double c2, s2;
};
constexpr int kTrigSlots = kMaxPartials;  // the reduction scratch: kMaxPartials * 32 bytes
constexpr unsigned long long kBusy = 1ull, kAcos = 1ull << 63;

__device__ __forceinline__ unsigned long long load_acquire(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

// cos^2 and sin^2 of an angle; what 0: atan(b / a); 1: a itself; kAcos: acos(a / b).
__device__ __forceinline__ double2 squared_cosines(unsigned long long what, double a, double b) {
    const double th = what == 0 ? atan(b / a) : what == kAcos ? acos(a / b) : a;
    const double c = cos(th), sn = sin(th);
    return make_double2(c * c, sn * sn);
}

// squared_cosines from the table, or into it.
// a is never the pattern of 0 or kBusy, which mark a slot without values: it is
// 1e-10 or more as a coordinate difference, and an angle given itself is that of
// ady >= 1e-10 > adx or a right one.
__device__ __forceinline__ double2 trig2(TrigSlot* __restrict__ table, unsigned long long what, double a, double b) {
    const unsigned long long ka = (unsigned long long)__double_as_longlong(a) ^ (what == kAcos ? kAcos : 0ull),
                             kb = (unsigned long long)__double_as_longlong(b) + what;
    unsigned h = (unsigned)(((ka ^ (kb * 0xD6E8FEB86659FD93ull)) * 0x9E3779B97F4A7C15ull) >> 40) % kTrigSlots;
    TrigSlot* mine = nullptr;
    for (int probe = 0; probe < 4; probe++, h = (h + 1) % kTrigSlots) {
        TrigSlot* s = table + h;
        unsigned long long k = load_acquire(&s->ka);
        if (k == ka && s->kb == kb) return make_double2(s->c2, s->s2);
        if (k == 0 && (k = atomicCAS(&s->ka, 0ull, kBusy)) == 0) {
            mine = s;
            break;
        }
    }
    const double2 r = squared_cosines(what, a, b);
    if (mine) {
        mine->kb = kb;
        mine->c2 = r.x;
        mine->s2 = r.y;
        __threadfence();
        atomicExch(&mine->ka, ka);
    }
    return r;
}

// scr of the bond between i and c of length L0 (kernel_cal_surf_coff_F,
// Surf_Corr.cu:160-232); trig gives an angle's squared cosines (squared_cosines).
template <class Trig>
__device__ __forceinline__ double surface_coefficient(const KParams& P, const double* __restrict__ x,
                                                      const double* __restrict__ y, const double* __restrict__ z,
                                                      const double* __restrict__ fnx, const double* __restrict__ fny,
                                                      const double* __restrict__ fnz, int64_t i, int64_t c, double L0,
                                                      const Trig& trig) {
    const double half_pi = 90.0 * P.pi / 180.0;
    const double scx = (fnx[i] + fnx[c]) / 2.0;
    const double scy = (fny[i] + fny[c]) / 2.0;
    const double adx = fabs(x[c] - x[i]), ady = fabs(y[c] - y[i]);
    // one call of trig for each angle, whatever its case: the lanes of a warp on a
    // lattice hold all of them
    const double2 none = make_double2(1.0, 0.0);  // cos(0), sin(0)
    if (P.dim == 2) {
        const bool upright = adx <= 1.0e-10;
        const double2 t =
            ady > 1.0e-10 ? trig(upright ? 1ull : 0ull, upright ? half_pi : adx, upright ? 0.0 : ady) : none;
        return sqrt(1.0 / (t.x / (scx * scx) + t.y / (scy * scy)));
    }
    const double scz = (fnz[i] + fnz[c]) / 2.0;
    const double adz = fabs(z[c] - z[i]);
    const bool flat = adz < 1.0e-10, upright = adx < 1.0e-10;
    if (!flat && upright && ady < 1.0e-10) return scz;
    // (not flat and upright: adx may be zero, atan of an infinite quotient, and ady is 1e-10 or more)
    const double up = upright && !flat ? atan(ady / adx) : half_pi;
    const double2 t = flat && !(ady >= 1.0e-10)
                          ? none
                          : trig(upright ? 1ull : 0ull, upright ? up : adx, upright ? 0.0 : ady);
    const double2 p = trig(flat ? 1ull : kAcos, flat ? half_pi : adz, flat ? 0.0 : L0);
    return sqrt(1.0 / (t.x / (scx * scx) + t.y / (scy * scy) + p.x / (scz * scz)));
}

// scr per bond.  The coefficient is the same, bit for bit, from both ends (sums
// of two and absolute differences), so one thread per row forms the bonds to
// higher neighbours and writes both directions; the other one is at the mirrored
// position of an interior row, searched for elsewhere.  7.0M bonds: 2.0 ms with a
// warp per row, 0.55 so.
__global__ void __launch_bounds__(128) k_surface_coeff(KParams P, const double* __restrict__ x, const double* __restrict__ y,
                                const double* __restrict__ z, const int64_t* __restrict__ rowptr,
                                const int* __restrict__ NL, const double* __restrict__ idist,
                                const double* __restrict__ fnx, const double* __restrict__ fny,
                                const double* __restrict__ fnz, TrigSlot* __restrict__ table,
                                double* __restrict__ scr) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= P.N) return;
    const auto trig = [table](unsigned long long what, double a, double b) { return trig2(table, what, a, b); };
    const int64_t q0 = rowptr[i], q1 = rowptr[i + 1];
    int64_t q = q0;
    for (int64_t hi = q1; q < hi;) {  // the first neighbour above i
        const int64_t mid = (q + hi) / 2;
        if (NL[mid] > i)
            hi = mid;
        else
            q = mid + 1;
    }
    for (; q < q1; q++) {
        const int64_t c = NL[q];
        const double v = surface_coefficient(P, x, y, z, fnx, fny, fnz, i, c, idist[q], trig);
        scr[q] = v;
        // the same bond in row c
        const int64_t c0 = rowptr[c], c1 = rowptr[c + 1];
        int64_t m = c1 - 1 - (q - q0);
        if (m < c0 || NL[m] != i) {
            m = c0;
            for (int64_t hi = c1; m < hi;) {
                const int64_t mid = (m + hi) / 2;
                if (NL[mid] >= i)
                    hi = mid;
                else
                    m = mid + 1;
            }
        }
        if (m < c1 && NL[m] == i) scr[m] = v;  // (every bond has its mirror)
    }
}

// Rows an SM up to which the surface coefficient (and the pre-crack pass) takes a
// warp per row: a thread's bonds come one after the other, most of their angles
// not yet in the table.  surface_correct as a whole, us, thread / warp per row here
// (152 SMs): 2-D 100 rows 149 / 36, 3,600 147 / 73, 10,000 204 / 187, off the
// lattice 196 / 165; 3-D 216 rows 852 / 130, 5,184 945 / 564, 10,800 1,126 / 1,073,
// off the lattice 5,184 944 / 427.  Beyond, the table wins on a lattice (2-D 22,500
// rows 303 us, 401 by a warp per row; 3-D 32,400 1,821, 3,334).
constexpr int kWarpRowsPerSm = 72;

// scr per bond, one warp per row and every bond's angles by itself: for the few
// rows of a small specimen (kWarpRowsPerSm).
__global__ void __launch_bounds__(256) k_surface_coeff_warp(KParams P, const double* __restrict__ x,
                                const double* __restrict__ y, const double* __restrict__ z,
                                const int64_t* __restrict__ rowptr, const int* __restrict__ NL,
                                const double* __restrict__ idist, const double* __restrict__ fnx,
                                const double* __restrict__ fny, const double* __restrict__ fnz,
                                double* __restrict__ scr) {
    const int64_t i = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    if (i >= P.N) return;
    const int64_t q1 = rowptr[i + 1];
    for (int64_t q = rowptr[i] + (threadIdx.x & 31); q < q1; q += 32)
        scr[q] = surface_coefficient(P, x, y, z, fnx, fny, fnz, i, NL[q], idist[q], squared_cosines);
}

// Pre-crack segment test (Base_Function.cu:39-81) on nodes [r0, r1)
// (the reference tests [0, N_int); a batch cracks one specimen at a time).
// LANES threads per row: one, or a warp's 32 up to kWarpRowsPerSm rows an SM, where
// a row's bonds one after the other would be the time of the pass (us, a thread /
// a warp per row, crack at 0.3 rad along the plate: 100 rows 48 / 13, 3,600 58 / 15,
// 10,000 52 / 28, 14,400 44 / 34, 22,500 44 / 44, 40,000 44 / 69; upright ones 13 /
// 7, 15 / 9, 15 / 15, 15 / 21, 15 / 27, 15 / 45).  A bond is cut when
// both ends lie within the segment's length and on different sides of its line,
// so a row fails all its bonds' tests at once when its own end does not, or when
// it is further from the line than a bond reaches (reach: an upper bound of
// |side_c - side_i| over a family of horizon delta, with room for rounding;
// infinite where the coordinates may have been written since the family was
// built).  Only the rows along the segment, about seven in a plate's height, walk
// their bonds; the whole test per bond spent the FP64 pipe's time on the others
// (7.0M bonds: 1.65 ms).
template <int LANES>
__global__ void k_set_crack_2d(KParams P, double delta, int64_t r0, int64_t r1, double clength, double lx, double ly,
                               double theta, const double* __restrict__ x, const double* __restrict__ y,
                               const int64_t* __restrict__ rowptr, const int* __restrict__ NL,
                               int* __restrict__ fail) {
    __shared__ double sk[3];  // the angle's functions, once per block
    if (threadIdx.x == 0) {
        const double t = tan(theta);
        sk[0] = t;
        sk[1] = sqrt(1 + t * t);
        sk[2] = clength * sin(theta) / 2.0;
    }
    __syncthreads();
    const int64_t i = r0 + (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / LANES;
    const int lane = threadIdx.x % LANES;
    if (i >= r1) return;
    const double xi = x[i], yi = y[i];
    if (fabs(theta - P.pi / 2.0) < 0.0001) {
        const double half = sk[2];
        if (!(fabs(yi - ly) < half) || fabs(xi - lx) > 1.001 * delta) return;
        for (int64_t q = rowptr[i] + lane; q < rowptr[i + 1]; q += LANES) {
            const int64_t c = NL[q];
            if (fabs(y[c] - ly) < half && (x[c] - lx) * (xi - lx) < 0.0) fail[q] = 0;
        }
        return;
    }
    const double t = sk[0], norm = sk[1];
    // a node's distance along the line from the segment's centre
    auto along = [&](double xa, double ya) {
        const double dist = (ya - ly) * (ya - ly) + (xa - lx) * (xa - lx);
        const double v = (t * xa - ya - lx * t + ly) / norm;
        return sqrt(dist - v * v);
    };
    auto side = [&](double xa, double ya) { return t * xa - lx * t + ly - ya; };
    const double bi = side(xi, yi);
    const double reach = 1.001 * delta * (1.0 + fabs(t)) + 1e-12 * (fabs(t * xi) + fabs(t * lx) + fabs(ly) + fabs(yi));
    if (fabs(bi) > reach || !(along(xi, yi) < clength / 2.0)) return;
    for (int64_t q = rowptr[i] + lane; q < rowptr[i + 1]; q += LANES) {
        const int64_t c = NL[q];
        if (side(x[c], y[c]) * bi <= 0 && along(x[c], y[c]) < clength / 2.0) fail[q] = 0;
    }
}

// Notch cut of the Kalthoff-Winkler slab (Solve_Kalthoff_Winkler.cu:40-63).
__global__ void k_set_crack_kw(KParams P, double rad, const double* __restrict__ x, const double* __restrict__ y,
                               const int64_t* __restrict__ rowptr, const int* __restrict__ NL,
                               int* __restrict__ fail) {
    const int64_t i = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (i >= P.N_int) return;
    for (int64_t q = rowptr[i] + lane; q < rowptr[i + 1]; q += 32) {
        const int64_t c = NL[q];
        const bool upper = (y[c] >= -1.0e-10) | (y[i] >= -1.0e-10);
        if (((x[c] > -rad && x[i] < -rad) | (x[i] > -rad && x[c] < -rad)) && upper) fail[q] = 0;
        if (((x[c] > rad && x[i] < rad) | (x[i] > rad && x[c] < rad)) && upper) fail[q] = 0;
    }
}

// ---- SELL-32 layout -------------------------------------------------------

__global__ void k_slice_width(int64_t N, int64_t nslices, const int* __restrict__ NN, int* __restrict__ width) {
    const int64_t s = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (s >= nslices) return;
    const int64_t r = s * 32 + lane;
    int v = r < N ? NN[r] : 0;
    for (int off = 16; off > 0; off >>= 1) v = max(v, __shfl_down_sync(0xffffffffu, v, off));
    if (lane == 0) width[s] = v;
}

// The reference vector xa rounded to float per component (xf, z = 0 in 2-D)
// and the exact constant |xf|^2 - l0^2 as a float pair (c0): products of
// floats are exact doubles, and the sums are carried as double pairs
// (TwoSum / FMA TwoProduct); sh - ph is exact, both within a factor 2 of
// l0^2.  l0 itself as a float pair (lf).
__device__ void float_reference(const double xa[3], int dim, double L0, float xf[3], float2& c0, float2& lf) {
    double sh = 0.0, sl = 0.0;
    xf[2] = 0.0f;
    for (int a = 0; a < dim; a++) {
        const float f = __double2float_rn(xa[a]);
        xf[a] = f;
        const double sq = (double)f * (double)f;  // exact: 24-bit x 24-bit mantissas
        const double t = sh + sq;
        const double bb = t - sh;
        sl += (sh - (t - bb)) + (sq - bb);
        sh = t;
    }
    const double ph = L0 * L0;
    const double pl = fma(L0, L0, -ph);
    const ff cf = ff_split((sh - ph) + (sl - pl));
    c0 = make_float2(cf.h, cf.l);
    const ff l = ff_split(L0);
    lf = make_float2(l.h, l.l);
}

// The CSR index of every slot (-1: padding), one warp per slice with a row per
// lane.
__global__ void k_sell_csr(int64_t N, int64_t nslices, const int* __restrict__ width, const int64_t* __restrict__ base,
                           const int* __restrict__ NN, const int64_t* __restrict__ rowptr, int* __restrict__ csr) {
    const int64_t s = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (s >= nslices) return;
    const int64_t r = s * 32 + lane;
    const int nn = r < N ? NN[r] : 0, q0 = r < N ? (int)rowptr[r] : 0, W = width[s];
    int* out = csr + base[s] + lane;
    for (int k = 0; k < W; k++) out[(int64_t)k * 32] = k < nn ? q0 + k : -1;
}

// The general layout's records, one thread per slot.  Padding slots point at
// their own row, carry zero coefficients and a cleared intact bit, so they
// contribute nothing.
__global__ void k_sell_fill(KParams P, int64_t nslices, const int* __restrict__ width,
                            const int64_t* __restrict__ base, const int* __restrict__ NN,
                            const int64_t* __restrict__ rowptr, const int* __restrict__ NL,
                            const double* __restrict__ x, const double* __restrict__ y, const double* __restrict__ z,
                            const double* __restrict__ idist, const double* __restrict__ fac,
                            const double* __restrict__ scr, const double* __restrict__ w, const double* __restrict__ m,
                            const double* __restrict__ node_bc, const double* __restrict__ node_s0, Sell S) {
    const int64_t s = blockIdx.y * (int64_t)gridDim.x + blockIdx.x;
    if (s >= nslices) return;
    const int W = width[s];
    const int64_t b = base[s];
    for (int t = threadIdx.x; t < W * 32; t += blockDim.x) {
        const int k = t >> 5, l = t & 31;
        const int64_t r = s * 32 + l;
        const int64_t slot = b + t;
        const bool used = r < P.N && k < NN[r];
        const int64_t q = used ? rowptr[r] + k : -1;
        if (!used) {
            if (S.rec) {
                BondRec R;
                R.col = (int)(r < P.N ? r : 0);
                R.xf[0] = R.xf[1] = R.xf[2] = 0.0f;
                R.c0 = make_float2(0.0f, 0.0f);
                R.l0 = make_float2(1.0f, 0.0f);
                R.k2 = make_float2(0.0f, 0.0f);
                R.ecrit = HUGE_VAL;
                S.rec[slot] = R;
            }
            if (S.sgeo) {
                StateGeo G{};
                G.col = (int)(r < P.N ? r : 0);
                G.l0 = make_float2(1.0f, 0.0f);
                S.sgeo[slot] = G;
                S.sth[slot] = StateTheta{};
                StateForce F{};
                F.ecrit = HUGE_VAL;
                S.sfo[slot] = F;
                S.e[slot] = make_float2(0.0f, 0.0f);
            }
            continue;
        }
        const int64_t c = NL[q];
        const double L0 = idist[q];
        // break when s = (L - L0)/L0 > s0, i.e. e = L - L0 > s0 L0; the 3-D
        // kernels break only bonds whose ends both have y >= -0.04 (Force_Bond.cu:117)
        bool breakable = true;
        if (P.dim == 3) breakable = y[r] >= P.break_ymin && y[c] >= P.break_ymin;
        // a batch of specimens carries bc and s0 per node (the row's specimen)
        const double s0 = node_s0 ? node_s0[r] : P.critical_s;
        const double bc = node_bc ? node_bc[r] : P.bc;
        const double ecrit = breakable ? s0 * L0 : HUGE_VAL;
        if (S.rec) {
            const double k2 = 2.0 * (P.vol * fac[q] * bc * scr[q]) / L0;
            BondRec R;
            R.col = (int)c;
            R.ecrit = ecrit;
            const ff kf = ff_split(k2 * S.kscale_inv);
            R.k2 = make_float2(kf.h, kf.l);
            const double xa[3] = {x[c] - x[r], y[c] - y[r], P.dim == 3 ? z[c] - z[r] : 0.0};
            float_reference(xa, P.dim, L0, R.xf, R.c0, R.l0);
            S.rec[slot] = R;
        }
        if (S.sgeo) {
            const double pr = P.pratio;
            double a_coef, b_coef, th_coef;
            if (P.dim == 2) {
                a_coef = (2.0 * pr - 1.0) / (pr - 1.0) * (2.0 * P.K - 32.0 * P.G / 9.0);
                b_coef = 8.0 * P.G;
                th_coef = 2.0 * (2.0 * pr - 1.0) / (pr - 1.0);
            } else {
                a_coef = 3.0 * P.K - 5.0 * P.G;  // 3K th w L0/m + 15G/m w (e - th L0/3)
                b_coef = 15.0 * P.G;
                th_coef = 3.0;
            }
            const double wf = w[q] * fac[q] * P.vol;
            StateTheta T;
            T.xi[0] = x[c] - x[r];
            T.xi[1] = y[c] - y[r];
            T.xi[2] = P.dim == 3 ? z[c] - z[r] : 0.0;
            // the coefficients as float pairs, scaled by powers of two (exact)
            const ff cth = ff_split(th_coef * w[q] * L0 * fac[q] * P.vol * ldexp(1.0, S.sth_exp));
            T.cth = make_float2(cth.h, cth.l);
            StateGeo G;
            G.col = (int)c;
            float_reference(T.xi, P.dim, L0, G.xf, G.c0, G.l0);
            StateForce F;
            const double cs = ldexp(1.0, S.sn_exp - S.st_exp);
            const ff c1 = ff_split(2.0 * a_coef * wf * L0 * cs), c2 = ff_split(2.0 * b_coef * wf * cs);
            F.c1 = make_float2(c1.h, c1.l);
            F.c2 = make_float2(c2.h, c2.l);
            F.ecrit = ecrit;
            F.xiz = T.xi[2];
            S.sgeo[slot] = G;
            S.sth[slot] = T;
            S.sfo[slot] = F;
            S.e[slot] = make_float2(0.0f, 0.0f);
        }
    }
}

// ---- compact layout of the 2-D bond-based kernels ---------------------------
//
// Offset classes: the bonds of one specimen whose reference vectors round to
// the same float vector xf (on a lattice, one class per lattice offset).  A
// hash table in device memory, one region of kRegion slots per specimen (a
// single plate is one specimen), collects the classes with the smallest bond
// length of each (l0t); the host numbers them per specimen in key order
// (deterministic, and the same for a plate alone and inside a batch) and
// builds one template per class; each slot then stores dl = l0 - l0t, the
// class id and k2 / 2 in a 16-byte record (bondtpl.h).

constexpr int kRegion = 256;  // hash slots per specimen (power of two)
constexpr unsigned long long kEmptyKey = ~0ull;

__device__ __forceinline__ unsigned long long class_key(double xa, double ya) {
    return ((unsigned long long)__float_as_uint(__double2float_rn(xa)) << 32) |
           (unsigned long long)__float_as_uint(__double2float_rn(ya));
}
__device__ __forceinline__ unsigned class_hash(unsigned long long k) {
    return (unsigned)((k * 0x9E3779B97F4A7C15ull) >> 56);  // 8 bits
}
// 3-D: a 64-bit mix of the three float components.  Not injective: the
// inserting thread stores its float vector beside the key, and the record
// fill checks every member's vector against its class's (a collision makes
// the layout unsupported, never a wrong class).
__device__ __forceinline__ unsigned long long class_key3(double xa, double ya, double za) {
    unsigned long long k = ((unsigned long long)__float_as_uint(__double2float_rn(xa)) << 32) |
                           (unsigned long long)__float_as_uint(__double2float_rn(ya));
    k ^= (unsigned long long)__float_as_uint(__double2float_rn(za)) * 0xD6E8FEB86659FD93ull;
    k ^= k >> 31;
    k *= 0xBF58476D1CE4E5B9ull;
    k ^= k >> 29;
    return k == kEmptyKey ? 0ull : k;
}

// z null: 2-D keys (the float vector itself); otherwise 3-D keys, and the
// thread that inserts a key writes its float vector into vec.  A thread per row,
// so that the lanes of a warp mostly look at one class at a time.
__global__ void k_class_insert(int64_t N, const int* __restrict__ NN,
                               const int64_t* __restrict__ rowptr, const int* __restrict__ NL,
                               const int* __restrict__ grp, const double* __restrict__ x,
                               const double* __restrict__ y, const double* __restrict__ z,
                               const double* __restrict__ idist, unsigned long long* __restrict__ keys,
                               unsigned long long* __restrict__ l0min, float4* __restrict__ vec,
                               int* __restrict__ overflow) {
    const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (r >= N) return;
    const int64_t q0 = rowptr[r];
    const int nn = NN[r];
    const int64_t region = grp ? grp[r] : 0;
    const double xr = x[r], yr = y[r], zr = z ? z[r] : 0.0;
    for (int k = 0; k < nn; k++) {
        const int64_t q = q0 + k, c = NL[q];
        const double xa = x[c] - xr, ya = y[c] - yr, za = z ? z[c] - zr : 0.0;
        const unsigned long long key = z ? class_key3(xa, ya, za) : class_key(xa, ya);
        const unsigned long long lb = (unsigned long long)__double_as_longlong(idist[q]);
        unsigned h = class_hash(key);
        bool done = false;
        for (int probe = 0; probe < kRegion && !done; probe++, h = (h + 1) & (kRegion - 1)) {
            const int64_t i = region * kRegion + h;
            // off the lattice a table is full at once, and every bond after that would
            // look through all of it, a row's one after the other (900 nodes in 3-D:
            // the whole set-up 7.7 ms, 0.8 with the flag looked at; a lattice's runs
            // are shorter than this)
            if (probe == 32 && __ldcg(overflow)) return;
            // looked at before it is swapped: after the first few bonds of a
            // class both words only have to be read, and the atomics of all
            // bonds on a few dozen addresses took 1.43 ms at 7.0M bonds
            unsigned long long prev = __ldcg(keys + i);
            if (prev == kEmptyKey) prev = atomicCAS(keys + i, kEmptyKey, key);
            if (prev == kEmptyKey || prev == key) {
                if (lb < __ldcg(l0min + i)) atomicMin(l0min + i, lb);  // positive doubles order like their bit patterns
                if (prev == kEmptyKey && vec)
                    vec[i] = make_float4(__double2float_rn(xa), __double2float_rn(ya), __double2float_rn(za), 0.0f);
                done = true;
            }
        }
        if (!done) atomicExch(overflow, 1);
    }
}

// Records of the compact layout; *bad is set where a slot cannot be
// represented (dl not a float with a free low byte).  One warp per slice with
// a row per lane.  What does not have to run on the FP64 pipe does not (22
// FP64 instructions a bond took 0.28 ms at 7.0M bonds): the length's difference
// from its class comes from the bit patterns, a volume factor of one is left
// out, and the powers of two of k2 = 2 (vol fac bc scr) / l0 times the scale go
// into the exponent (exact, like the products they replace).
__global__ void k_rec16_fill(KParams P, int64_t nslices, const int* __restrict__ width,
                             const int64_t* __restrict__ base, const int* __restrict__ NN,
                             const int64_t* __restrict__ rowptr, const int* __restrict__ NL,
                             const int* __restrict__ grp, const double* __restrict__ x, const double* __restrict__ y,
                             const double* __restrict__ idist, const double* __restrict__ fac,
                             const double* __restrict__ scr, const double* __restrict__ node_bc,
                             const unsigned long long* __restrict__ keys, const int* __restrict__ ids,
                             const int* __restrict__ inst_tbase, const bt::Tpl* __restrict__ tpl, int k2exp,
                             bt::Rec* __restrict__ rec, int* __restrict__ bad) {
    const int64_t s = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (s >= nslices) return;
    const int64_t r = s * 32 + lane;
    const bool row = r < P.N;
    const int W = width[s], nn = row ? NN[r] : 0;
    const int64_t q0 = row ? rowptr[r] : 0;
    const double xr = row ? x[r] : 0.0, yr = row ? y[r] : 0.0;
    const int64_t region = grp && nn > 0 ? grp[r] : 0;
    const int64_t tb = inst_tbase ? inst_tbase[region] : 0;
    const double bc = node_bc && row ? node_bc[r] : P.bc;
    const double vb = P.vol * bc;
    bt::Rec* out = rec + base[s] + lane;
    for (int k = 0; k < W; k++) {
        bt::Rec R;
        if (k >= nn) {
            R.col = row ? (int)r : 0;
            R.dl = 0.0f;  // class 0, zero coefficient: a padding slot contributes nothing
            R.k2h = R.k2l = 0.0f;
            out[(int64_t)k * 32] = R;
            continue;
        }
        const int64_t q = q0 + k, c = NL[q];
        const unsigned long long key = class_key(x[c] - xr, y[c] - yr);
        unsigned h = class_hash(key);
        int id = -1;
        for (int probe = 0; probe < kRegion; probe++, h = (h + 1) & (kRegion - 1)) {
            const int64_t i = region * kRegion + h;
            if (keys[i] == key) {
                id = ids[i];
                break;
            }
            if (keys[i] == kEmptyKey) break;
        }
        const double L0 = idist[q];
        float dl = 0.0f;
        bool fail = id < 0 || id > 255;
        if (!fail) {
            // l0 - l0t: in one binade the difference of the patterns in ulps
            const unsigned long long lb = (unsigned long long)__double_as_longlong(L0),
                                     tl = (unsigned long long)__double_as_longlong(tpl[tb + id].l0d);
            const unsigned long long ulps = lb - tl;  // l0t is the class's smallest length
            const int e = (int)(lb >> 52) - 1075 + 127;
            if ((lb >> 52) == (tl >> 52) && ulps < (1ull << 24) && e > 0 && e < 255) {
                dl = __uint2float_rn((unsigned)ulps) * __uint_as_float((unsigned)e << 23);
            } else {
                const double dlv = L0 - tpl[tb + id].l0d;  // exact: l0 and l0t within a factor two
                dl = __double2float_rn(dlv);
                fail = (double)dl != dlv;
            }
        }
        const unsigned dlb = __float_as_uint(dl);
        if (fail || (dlb & 0xffu) != 0u) atomicExch(bad, 1);
        R.col = (int)c;
        R.dl = __uint_as_float((dlb & ~0xffu) | (unsigned)(id & 0xff));
        const double f = fac[q];
        const double a = __double_as_longlong(f) == __double_as_longlong(1.0) ? vb : P.vol * f * bc;
        const double k1 = (a * scr[q]) / L0;
        const long long kb = __double_as_longlong(k1);
        const int ke = (int)(kb >> 52) & 0x7ff;
        const double k2 = ke > 100 && ke < 1900 && k2exp > -100 && k2exp < 100
                              ? __longlong_as_double(kb + ((long long)k2exp << 52))
                              : k1 * ldexp(1.0, k2exp);
        const ff kf = ff_split(k2);
        R.k2h = kf.h;
        R.k2l = kf.l;
        out[(int64_t)k * 32] = R;
    }
}

// The coefficients of one state-based bond (the state records of
// k_sell_fill), with the context's power-of-two scales, in doubles.
__device__ __forceinline__ void state_coefs(const KParams& P, double L0, double w, double fac, int sn_exp,
                                            int sth_exp, int st_exp, double& cth, double& c1, double& c2) {
    const double pr = P.pratio;
    double a_coef, b_coef, th_coef;
    if (P.dim == 2) {
        a_coef = (2.0 * pr - 1.0) / (pr - 1.0) * (2.0 * P.K - 32.0 * P.G / 9.0);
        b_coef = 8.0 * P.G;
        th_coef = 2.0 * (2.0 * pr - 1.0) / (pr - 1.0);
    } else {
        a_coef = 3.0 * P.K - 5.0 * P.G;  // 3K th w L0/m + 15G/m w (e - th L0/3)
        b_coef = 15.0 * P.G;
        th_coef = 3.0;
    }
    const double wf = w * fac * P.vol;
    cth = th_coef * w * L0 * fac * P.vol * ldexp(1.0, sth_exp);
    const double cs = ldexp(1.0, sn_exp - st_exp);
    c1 = 2.0 * a_coef * wf * L0 * cs;
    c2 = 2.0 * b_coef * wf * cs;
}

// Records of the 3-D bond-based compact layout: {column, dl with the class
// id, k2 / 2 as a pair}, the pair negated where the bond may not break (an
// end below y = -0.04, Force_Bond.cu:117).  *bad as in k_rec16_fill, and also
// where a slot's float vector is not its class's (a key collision).
__global__ void k_rec16_fill3(KParams P, int64_t nslices, const int* __restrict__ width,
                              const int64_t* __restrict__ base, const int* __restrict__ csr,
                              const int* __restrict__ NL, const double* __restrict__ x, const double* __restrict__ y,
                              const double* __restrict__ z, const double* __restrict__ idist,
                              const double* __restrict__ fac, const double* __restrict__ scr,
                              const unsigned long long* __restrict__ keys, const int* __restrict__ ids,
                              const bt::Tpl3* __restrict__ tpl, double kscale_half_inv, bt::Rec* __restrict__ rec,
                              int* __restrict__ bad) {
    const int64_t s = blockIdx.y * (int64_t)gridDim.x + blockIdx.x;
    if (s >= nslices) return;
    const int W = width[s];
    const int64_t b = base[s];
    for (int t = threadIdx.x; t < W * 32; t += blockDim.x) {
        const int64_t slot = b + t;
        const int q = csr[slot];
        const int64_t r = s * 32 + (t & 31);
        bt::Rec R;
        if (q < 0) {
            R.col = (int)(r < P.N ? r : 0);
            R.dl = 0.0f;  // class 0, zero coefficient: a padding slot contributes nothing
            R.k2h = R.k2l = 0.0f;
            rec[slot] = R;
            continue;
        }
        const int64_t c = NL[q];
        const double xv[3] = {x[c] - x[r], y[c] - y[r], z[c] - z[r]};
        const unsigned long long key = class_key3(xv[0], xv[1], xv[2]);
        unsigned h = class_hash(key);
        int id = -1;
        for (int probe = 0; probe < kRegion; probe++, h = (h + 1) & (kRegion - 1)) {
            if (keys[h] == key) {
                id = ids[h];
                break;
            }
            if (keys[h] == kEmptyKey) break;
        }
        bool fail = id < 0 || id > 255;
        const double L0 = idist[q];
        double dlv = 0.0;
        if (!fail) {
            const bt::Tpl3& T = tpl[id];
            dlv = L0 - T.l0d;
            for (int a = 0; a < 3; a++)
                if (__double2float_rn(xv[a]) != T.xf[a]) fail = true;  // another vector under the same key
        }
        const float dl = __double2float_rn(dlv);
        const unsigned dlb = __float_as_uint(dl);
        if ((double)dl != dlv || (dlb & 0xffu) != 0u) fail = true;
        if (fail) atomicExch(bad, 1);
        R.col = (int)c;
        R.dl = __uint_as_float((dlb & ~0xffu) | (unsigned)(id & 0xff));
        const double k2 = 2.0 * (P.vol * fac[q] * P.bc * scr[q]) / L0;
        const ff kf = ff_split(k2 * kscale_half_inv);
        const bool breakable = y[r] >= P.break_ymin && y[c] >= P.break_ymin;
        R.k2h = breakable ? kf.h : -kf.h;
        R.k2l = breakable ? kf.l : -kf.l;
        rec[slot] = R;
    }
}

// A component of a reference vector x_c - x_i (as the reference rounds it,
// Force_State.cu:71-72) not within 2^31 representable doubles of its float
// rounding, which is its class's, or of another sign: only where that is zero or
// subnormal.  Such a problem takes the records layout, as one whose slots cannot
// hold the distance does.
__device__ __forceinline__ bool far_from_class(double v) {
    const long long xb = __double_as_longlong((double)__double2float_rn(v)), vb = __double_as_longlong(v);
    return (vb < 0) != (xb < 0) || vb - xb < INT_MIN || vb - xb > INT_MAX;
}

// Records of the 2-D state-based compact layout: rec8 = {column, dl with the
// class id}.  A slot whose bond has the class's reference length (dl = 0; every
// class has one) writes the class's coefficients into stpl (such slots compute
// identical values).  *bad as in k_rec16_fill, and also where a reference
// vector is far from its class's.
__global__ void k_state_compact_fill(KParams P, int64_t nslices, const int* __restrict__ width,
                                     const int64_t* __restrict__ base, const int* __restrict__ csr,
                                     const int* __restrict__ NL, const double* __restrict__ x,
                                     const double* __restrict__ y, const double* __restrict__ idist,
                                     const double* __restrict__ fac, const double* __restrict__ w,
                                     const unsigned long long* __restrict__ keys, const int* __restrict__ ids,
                                     const bt::Tpl* __restrict__ tpl, int sn_exp, int sth_exp, int st_exp,
                                     int2* __restrict__ rec8, StateTpl* __restrict__ stpl,
                                     int* __restrict__ bad) {
    const int64_t s = blockIdx.y * (int64_t)gridDim.x + blockIdx.x;
    if (s >= nslices) return;
    const int W = width[s];
    const int64_t b = base[s];
    for (int t = threadIdx.x; t < W * 32; t += blockDim.x) {
        const int64_t slot = b + t;
        const int q = csr[slot];
        const int64_t r = s * 32 + (t & 31);
        if (q < 0) {
            rec8[slot] = make_int2((int)(r < P.N ? r : 0), 0);
            continue;
        }
        const int64_t c = NL[q];
        const double xa = x[c] - x[r], ya = y[c] - y[r];  // the reference's rounding (Force_State.cu:71-72)
        const unsigned long long key = class_key(xa, ya);
        unsigned h = class_hash(key);
        int id = -1;
        for (int probe = 0; probe < kRegion; probe++, h = (h + 1) & (kRegion - 1)) {
            if (keys[h] == key) {
                id = ids[h];
                break;
            }
            if (keys[h] == kEmptyKey) break;
        }
        const double L0 = idist[q];
        const double dlv = id >= 0 ? L0 - tpl[id].l0d : 0.0;
        const float dl = __double2float_rn(dlv);
        const unsigned dlb = __float_as_uint(dl);
        bool fail = id < 0 || id > 255 || (double)dl != dlv || (dlb & 0xffu) != 0u;
        if (!fail)
            fail = far_from_class(xa) || far_from_class(ya);
        if (fail) atomicExch(bad, 1);
        const int dlw = (int)((dlb & ~0xffu) | (unsigned)(id & 0xff));
        rec8[slot] = make_int2((int)c, dlw);
        if (!fail && dlv == 0.0) {
            double cth, c1, c2;
            state_coefs(P, L0, w[q], fac[q], sn_exp, sth_exp, st_exp, cth, c1, c2);
            const ff a = ff_split(c1), bb = ff_split(c2), t3 = ff_split(cth);
            StateTpl& T = stpl[id];  // g1, g2 come from the host
            T.c1h = a.h, T.c1l = a.l, T.c2h = bb.h, T.c2l = bb.l;
            T.cth_h = t3.h, T.cth_l = t3.l;
        }
    }
}

// Records of the 3-D state-based compact layout, as k_state_compact_fill.
// *bad also where a slot's float vector is not its class's (a key collision).
__global__ void k_state_compact3_fill(KParams P, int64_t nslices, const int* __restrict__ width,
                                      const int64_t* __restrict__ base, const int* __restrict__ csr,
                                      const int* __restrict__ NL, const double* __restrict__ x,
                                      const double* __restrict__ y, const double* __restrict__ z,
                                      const double* __restrict__ idist, const double* __restrict__ fac,
                                      const double* __restrict__ w, const unsigned long long* __restrict__ keys,
                                      const int* __restrict__ ids, const bt::Tpl3* __restrict__ tpl, int sn_exp,
                                      int sth_exp, int st_exp, int2* __restrict__ rec8,
                                      StateTpl* __restrict__ stpl, int* __restrict__ bad) {
    const int64_t s = blockIdx.y * (int64_t)gridDim.x + blockIdx.x;
    if (s >= nslices) return;
    const int W = width[s];
    const int64_t b = base[s];
    for (int t = threadIdx.x; t < W * 32; t += blockDim.x) {
        const int64_t slot = b + t;
        const int q = csr[slot];
        const int64_t r = s * 32 + (t & 31);
        if (q < 0) {
            rec8[slot] = make_int2((int)(r < P.N ? r : 0), 0);
            continue;
        }
        const int64_t c = NL[q];
        // the reference's roundings of the reference vector (Force_State.cu:217-219)
        const double xv[3] = {x[c] - x[r], y[c] - y[r], z[c] - z[r]};
        const unsigned long long key = class_key3(xv[0], xv[1], xv[2]);
        unsigned h = class_hash(key);
        int id = -1;
        for (int probe = 0; probe < kRegion; probe++, h = (h + 1) & (kRegion - 1)) {
            if (keys[h] == key) {
                id = ids[h];
                break;
            }
            if (keys[h] == kEmptyKey) break;
        }
        bool fail = id < 0 || id > 255;
        const double L0 = idist[q];
        double dlv = 0.0;
        if (!fail) {
            const bt::Tpl3& T = tpl[id];
            dlv = L0 - T.l0d;
            for (int a = 0; a < 3; a++) {
                if (__double2float_rn(xv[a]) != T.xf[a]) fail = true;  // another vector under the same key
                if (far_from_class(xv[a])) fail = true;
            }
        }
        const float dl = __double2float_rn(dlv);
        const unsigned dlb = __float_as_uint(dl);
        if ((double)dl != dlv || (dlb & 0xffu) != 0u) fail = true;
        if (fail) atomicExch(bad, 1);
        const int dlw = (int)((dlb & ~0xffu) | (unsigned)(id & 0xff));
        rec8[slot] = make_int2((int)c, dlw);
        if (!fail && dlv == 0.0) {
            double cth, c1, c2;
            state_coefs(P, L0, w[q], fac[q], sn_exp, sth_exp, st_exp, cth, c1, c2);
            const ff a = ff_split(c1), bb = ff_split(c2), t3 = ff_split(cth);
            StateTpl& T = stpl[id];  // g1, g2 come from the host
            T.c1h = a.h, T.c1l = a.l, T.c2h = bb.h, T.c2l = bb.l;
            T.cth_h = t3.h, T.cth_l = t3.l;
        }
    }
}

// The "may break" flags of the 3-D state-based bonds (both ends at y >= -0.04,
// Force_State.cu:283) as one bit word per (slice, slot), like the intact flags.
__global__ void k_break_bits(KParams P, int64_t nslices, const int* __restrict__ width,
                             const int64_t* __restrict__ base, const int64_t* __restrict__ fbase,
                             const int* __restrict__ csr, const double* __restrict__ y, const int2* __restrict__ rec8,
                             uint32_t* __restrict__ bbits) {
    const int64_t s = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (s >= nslices) return;
    const int W = width[s];
    const bool row = s * 32 + lane < P.N && y[s * 32 + lane] >= P.break_ymin;
    for (int k = 0; k < W; k++) {
        const int64_t slot = base[s] + (int64_t)k * 32 + lane;
        const uint32_t word = __ballot_sync(0xffffffffu, row && csr[slot] >= 0 && y[rec8[slot].x] >= P.break_ymin);
        if (lane == 0) bbits[fbase[s] + k] = word;
    }
}

// Every slot's coefficients against its class's moved to the slot's length
// (c (1 + g dl)): *bad where one differs from the bond's own by more than
// 2^-45 of it.
__global__ void k_state_compact_check(KParams P, int64_t nslices, const int* __restrict__ width,
                                      const int64_t* __restrict__ base, const int* __restrict__ csr,
                                      const double* __restrict__ idist, const double* __restrict__ fac,
                                      const double* __restrict__ w, const int2* __restrict__ rec8,
                                      const StateTpl* __restrict__ stpl, int sn_exp, int sth_exp, int st_exp,
                                      int* __restrict__ bad) {
    const int64_t s = blockIdx.y * (int64_t)gridDim.x + blockIdx.x;
    if (s >= nslices) return;
    const int W = width[s];
    const int64_t b = base[s];
    for (int t = threadIdx.x; t < W * 32; t += blockDim.x) {
        const int64_t slot = b + t;
        const int q = csr[slot];
        if (q < 0) continue;
        const unsigned dlb = (unsigned)rec8[slot].y;
        const StateTpl T = stpl[dlb & 0xffu];
        const double dl = (double)__uint_as_float(dlb & ~0xffu);
        double cth, c1, c2;
        state_coefs(P, idist[q], w[q], fac[q], sn_exp, sth_exp, st_exp, cth, c1, c2);
        const double tol = ldexp(1.0, -45);
        const double f1 = 1.0 + (double)T.g1 * dl, f2 = 1.0 + (double)T.g2 * dl;
        const double d1 = fabs(((double)T.c1h + (double)T.c1l) * f1 - c1);
        const double d2 = fabs(((double)T.c2h + (double)T.c2l) * f2 - c2);
        const double d3 = fabs(((double)T.cth_h + (double)T.cth_l) * f1 - cth);
        if (!(d1 <= tol * fabs(c1)) || !(d2 <= tol * fabs(c2)) || !(d3 <= tol * fabs(cth))) atomicExch(bad, 1);
    }
}

// Intact flags: CSR int32 <-> SELL bit words.
__global__ void k_bits_from_csr(int64_t nslices, const int* __restrict__ width, const int64_t* __restrict__ base,
                                const int64_t* __restrict__ fbase, const int* __restrict__ csr,
                                const int* __restrict__ fail, int64_t n_rows_breakable, uint32_t* __restrict__ bits) {
    const int64_t s = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (s >= nslices) return;
    const int W = width[s];
    for (int k = 0; k < W; k++) {
        const int64_t slot = base[s] + k * 32 + lane;
        const int q = csr[slot];
        // rows past N_int have no fail storage in the reference (Memory.cu:39):
        // their bonds count as intact
        const bool alive = q >= 0 && ((s * 32 + lane) >= n_rows_breakable || fail[q] == 1);
        const uint32_t word = __ballot_sync(0xffffffffu, alive);
        if (lane == 0) bits[fbase[s] + k] = word;
    }
}

__global__ void k_csr_from_bits(int64_t nslices, const int* __restrict__ width, const int64_t* __restrict__ base,
                                const int64_t* __restrict__ fbase, const int* __restrict__ csr,
                                const uint32_t* __restrict__ bits, int* __restrict__ fail) {
    const int64_t s = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (s >= nslices) return;
    const int W = width[s];
    for (int k = 0; k < W; k++) {
        const int64_t slot = base[s] + k * 32 + lane;
        const int q = csr[slot];
        if (q >= 0) fail[q] = (bits[fbase[s] + k] >> lane) & 1u;
    }
}

// 1/m per node (IEEE-rounded, the dilatation pass's divisor reciprocal) and
// the same times 2^-sn as a float pair (the force pass's operand).
__global__ void k_inv_m(int64_t N, const double* __restrict__ m, double sn_scale, double* __restrict__ inv,
                        float4* __restrict__ nab) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < N) {
        const double v = 1.0 / m[i];
        inv[i] = v;
        const ff p = ff_split(v * sn_scale);
        reinterpret_cast<float2*>(nab + i)[1] = make_float2(p.h, p.l);  // the second pair of {theta/m, 1/m}
    }
}

unsigned warps_grid(int64_t nwarps) { return (unsigned)((nwarps * 32 + 255) / 256); }

}  // namespace

// Whether the family pass takes a warp per row instead of a thread, by the rows an
// SM gets.  A thread's bonds come one after the other, about 1 us each, whatever
// the number of rows up to 128 an SM, and again for every 128 more; a warp's row
// costs the same everywhere.  In 3-D a thread per row writes its bonds' two or
// three doubles 122 places apart, which goes well while the arrays fit the
// second-level cache.  Microseconds, thread / warp (152 SMs):
//   2-D rows             900       10,000     14,400     25,600     57,600    250,000
//   idist and fac     30 / 6     31 / 19    31 / 25    43 / 42    58 / 88   347 / 367
//   with w            62 / 8     64 / 42    62 / 56   103 / 99  150 / 209   634 / 888
//   energies, scr   231 / 133  220 / 196  221 / 225  293 / 326  416 / 610  1,709 / 2,495
//   3-D rows             216       10,800     27,000     46,656     57,600     72,000    180,000
//   idist and fac   124 / 12   152 / 76 192 / 182  251 / 312  266 / 383  440 / 477 1,705 / 1,187
//   with w          256 / 19  284 / 142 420 / 343  590 / 590  642 / 724  970 / 907 2,635 / 2,255
//   energies, scr 1,429 / 838 1,391 / 1,105 1,862 / 1,744 2,396 / 2,528 2,529 / 2,972 3,085 / 3,578 6,855 / 8,339
// (the last line: surface_correct as a whole, scr by a thread per row).
template <int DIM, bool ENERGY, bool WEIGHT>
static bool family_by_warps(int64_t rows, int64_t sms) {
    if (DIM == 2) return rows <= (ENERGY ? 80 : 168) * sms;
    if (ENERGY) return rows <= 188 * sms;
    return rows <= (WEIGHT ? 310 : 190) * sms || rows > (WEIGHT ? 420 : 470) * sms;
}

// The family pass with the stages asked for (energy: the surface test
// fields; weight: w and m); idist and fac are always written.
template <int DIM, bool ENERGY, bool WEIGHT>
static void launch_family_setup(pd_ctx* c, const KParams& P, cudaStream_t s) {
    const double sedload = DIM == 3 ? 0.6 * P.emod * 1.0e-6 : 0.5 * P.emod / (1.0 - P.pratio * P.pratio) * 1.0e-6;
    const bool warps = family_by_warps<DIM, ENERGY, WEIGHT>(P.N, c->num_sms);
    auto kernel = warps ? k_family_setup_warp<DIM, ENERGY, WEIGHT> : k_family_setup<DIM, ENERGY, WEIGHT>;
    const int block = warps ? 256 : 128;
    const unsigned grid = warps ? warps_grid(P.N) : (unsigned)((P.N + 127) / 128);
    kernel<<<grid, block, 0, s>>>(
        P, sedload, c->batch.node_bc, c->batch.node_sed, c->nf[PD_F_X], c->nf[PD_F_Y], c->nf[PD_F_Z], c->rowptr, c->NL,
        c->idist, c->fac, c->nf[PD_F_FNCST_X], c->nf[PD_F_FNCST_Y], c->nf[PD_F_FNCST_Z], c->w, c->nf[PD_F_M]);
    c->launches++;
}
template <bool ENERGY, bool WEIGHT>
static void launch_family_setup(pd_ctx* c, const KParams& P, cudaStream_t s) {
    if (P.dim == 3)
        launch_family_setup<3, ENERGY, WEIGHT>(c, P, s);
    else
        launch_family_setup<2, ENERGY, WEIGHT>(c, P, s);
}

int vol_corr(pd_ctx* c, cudaStream_t s) {
    if (!c->family) return set_err(c, PD_ERR_STATE, "vol_corr needs the bond family");
    launch_family_setup<false, false>(c, kparams(c->p), s);
    c->volcorr = true;
    c->prepared = false;
    return cuda_err(c, cudaGetLastError(), "vol_corr");
}

// vol_Corr and the surface energies in one family pass, then the coefficient
// pass (scr of a bond needs both end nodes' fncst: a grid-wide dependency).
// A state-based context also gets w and m from the first pass.
int surface_correct(pd_ctx* c, cudaStream_t s) {
    if (!c->family) return set_err(c, PD_ERR_STATE, "surface_correct needs the bond family");
    const KParams P = kparams(c->p);
    const bool state = c->p.model == PD_MODEL_STATE;
    if (state)
        launch_family_setup<true, true>(c, P, s);
    else
        launch_family_setup<true, false>(c, P, s);
    double *X = c->nf[PD_F_X], *Y = c->nf[PD_F_Y], *Z = c->nf[PD_F_Z];
    const double *FX = c->nf[PD_F_FNCST_X], *FY = c->nf[PD_F_FNCST_Y], *FZ = c->nf[PD_F_FNCST_Z];
    if (P.N <= kWarpRowsPerSm * (int64_t)c->num_sms) {
        k_surface_coeff_warp<<<warps_grid(P.N), 256, 0, s>>>(P, X, Y, Z, c->rowptr, c->NL, c->idist, FX, FY, FZ, c->scr);
    } else {
        cudaMemsetAsync(c->partials, 0, (size_t)kTrigSlots * sizeof(TrigSlot), s);
        k_surface_coeff<<<(unsigned)((P.N + 127) / 128), 128, 0, s>>>(P, X, Y, Z, c->rowptr, c->NL, c->idist, FX, FY, FZ,
                                                                      reinterpret_cast<TrigSlot*>(c->partials), c->scr);
    }
    c->launches++;
    c->volcorr = c->surfcorr = true;
    c->weights = c->weights || state;
    c->prepared = false;
    return cuda_err(c, cudaGetLastError(), "surface_correct");
}

// w and m in the family pass, which also (re)writes idist and fac: after a
// vol_corr call the same values again, without one the call stands for both.
int initial_weight(pd_ctx* c, cudaStream_t s) {
    if (!c->family) return set_err(c, PD_ERR_STATE, "initial_weight needs the bond family");
    launch_family_setup<false, true>(c, kparams(c->p), s);
    c->volcorr = true;
    c->weights = true;
    c->prepared = false;
    return cuda_err(c, cudaGetLastError(), "initial_weight");
}

int sync_fail_to_csr(pd_ctx* c, cudaStream_t s) {
    if (c->csr_fail_current) return PD_OK;
    const Sell& S = c->sell;
    k_csr_from_bits<<<warps_grid(S.nslices), 256, 0, s>>>(S.nslices, S.width, S.base, S.fbase, S.csr, S.bits,
                                                           c->fail);
    c->launches++;
    c->csr_fail_current = true;
    return cuda_err(c, cudaGetLastError(), "fail flags to CSR");
}

int sync_fail_to_bits(pd_ctx* c, cudaStream_t s) {
    if (c->bits_current) return PD_OK;
    const Sell& S = c->sell;
    k_bits_from_csr<<<warps_grid(S.nslices), 256, 0, s>>>(S.nslices, S.width, S.base, S.fbase, S.csr, c->fail,
                                                           c->p.N_int, S.bits);
    c->launches++;
    c->bits_current = true;
    return cuda_err(c, cudaGetLastError(), "fail flags to bits");
}

int set_crack_2d_rows(pd_ctx* c, int64_t r0, int64_t r1, double clength, double lx, double ly, double theta,
                      cudaStream_t s) {
    if (!c->family) return set_err(c, PD_ERR_STATE, "set_crack needs the bond family");
    if (r0 < 0 || r1 > c->p.N || r0 > r1) return set_err(c, PD_ERR_ARG, "set_crack row range out of bounds");
    if (r0 == r1) return PD_OK;
    int rc = sync_fail_to_csr(c, s);
    if (rc) return rc;
    const KParams P = kparams(c->p);
    const bool warps = r1 - r0 <= kWarpRowsPerSm * (int64_t)c->num_sms;
    auto kernel = warps ? k_set_crack_2d<32> : k_set_crack_2d<1>;
    kernel<<<warps ? warps_grid(r1 - r0) : (unsigned)((r1 - r0 + 255) / 256), 256, 0, s>>>(
        P, c->fam_delta, r0, r1, clength, lx, ly, theta, c->nf[PD_F_X], c->nf[PD_F_Y], c->rowptr, c->NL, c->fail);
    c->launches++;
    c->bits_current = false;
    return cuda_err(c, cudaGetLastError(), "set_crack_2d");
}

int set_crack_2d(pd_ctx* c, double clength, double lx, double ly, double theta, cudaStream_t s) {
    return set_crack_2d_rows(c, 0, c->p.N_int, clength, lx, ly, theta, s);
}

int set_crack_kw(pd_ctx* c, double rad, cudaStream_t s) {
    if (!c->family) return set_err(c, PD_ERR_STATE, "set_crack needs the bond family");
    int rc = sync_fail_to_csr(c, s);
    if (rc) return rc;
    const KParams P = kparams(c->p);
    k_set_crack_kw<<<warps_grid(P.N_int), 256, 0, s>>>(P, rad, c->nf[PD_F_X], c->nf[PD_F_Y], c->rowptr, c->NL,
                                                        c->fail);
    c->launches++;
    c->bits_current = false;
    return cuda_err(c, cudaGetLastError(), "set_crack_kw");
}

static void free_sell(pd_ctx* c) {
    Sell& S = c->sell;
    DeviceBlocks& mem = c->blocks;
    mem.give(S.width);
    mem.give(S.base);
    mem.give(S.fbase);
    mem.give(S.csr);
    mem.give(S.rec);
    mem.give(S.sgeo);
    mem.give(S.sth);
    mem.give(S.sfo);
    mem.give(S.e);
    mem.give(S.bits);
    mem.give(S.rec16);
    mem.give(S.tpl);
    mem.give(S.inst_tbase);
    mem.give(S.srec8);
    mem.give(S.stpl);
    mem.give(S.tpl3);
    mem.give(S.bbits);
    S.ntpl = 0;
    S.nslices = S.S = S.F = 0;
}

void release_sell(pd_ctx* c) {
    drop_graphs(c);
    free_sell(c);
}

// The compact layout (S.csr filled): offset classes per specimen, their
// templates and the slot records, for 2-D bond-based problems (one specimen
// or a batch) and state-based problems in 2-D and 3-D.  Returns
// PD_ERR_UNSUPPORTED (arrays released) where the problem does not fit it:
// more than 255 classes in a specimen (or a region of the hash table full), a
// bond length that differs from its class's smallest by more than a float
// with a free low byte can hold, a reference vector too far from its class's
// float vector, a coefficient off its class's by more than 2^-45, or (3-D) a
// key shared by two float vectors.
int build_compact(pd_ctx* c, cudaStream_t s) {
    const KParams P = kparams(c->p);
    Sell& S = c->sell;
    const int* grp = c->batch.node_group;
    const int64_t regions = c->batch.count > 0 ? c->batch.count : 1;
    const int64_t tsize = regions * kRegion;
    const bool state = c->p.model == PD_MODEL_STATE;
    const bool d3 = c->p.dim == 3;
    unsigned long long *keys = nullptr, *l0min = nullptr;
    int *ids = nullptr, *flags = nullptr;
    float4* vec = nullptr;
    DeviceBlocks& mem = c->blocks;
    auto cleanup = [&]() {
        mem.give(keys);
        mem.give(l0min);
        mem.give(ids);
        mem.give(flags);
        mem.give(vec);
    };
    auto release = [&]() {
        mem.give(S.tpl);
        mem.give(S.rec16);
        mem.give(S.inst_tbase);
        mem.give(S.srec8);
        mem.give(S.stpl);
        mem.give(S.tpl3);
        mem.give(S.bbits);
        S.ntpl = 0;
    };
    if (!mem.take(keys, tsize * 8) || !mem.take(l0min, tsize * 8) || !mem.take(ids, tsize * 4) ||
        !mem.take(flags, 2 * 4) || (d3 && !mem.take(vec, tsize * sizeof(float4)))) {
        cleanup();
        return set_err(c, PD_ERR_NOMEM, "offset-class table");
    }
    cudaMemsetAsync(keys, 0xff, tsize * 8, s);
    cudaMemsetAsync(l0min, 0xff, tsize * 8, s);
    cudaMemsetAsync(flags, 0, 2 * 4, s);
    if (vec) cudaMemsetAsync(vec, 0, tsize * sizeof(float4), s);
    const unsigned gx = (unsigned)std::min<int64_t>(S.nslices, 65535);
    const unsigned gy = (unsigned)((S.nslices + gx - 1) / gx);
    k_class_insert<<<(unsigned)((P.N + 255) / 256), 256, 0, s>>>(P.N, c->NN, c->rowptr, c->NL, grp,
                                                                 c->nf[PD_F_X], c->nf[PD_F_Y],
                                                                 d3 ? c->nf[PD_F_Z] : nullptr, c->idist, keys, l0min,
                                                                 vec, flags);
    c->launches++;
    std::vector<unsigned long long> hk((size_t)tsize), hl((size_t)tsize);
    std::vector<float4> hv(d3 ? (size_t)tsize : 0);
    int hflags[2] = {0, 0};
    cudaMemcpyAsync(hk.data(), keys, tsize * 8, cudaMemcpyDeviceToHost, s);
    cudaMemcpyAsync(hl.data(), l0min, tsize * 8, cudaMemcpyDeviceToHost, s);
    if (d3) cudaMemcpyAsync(hv.data(), vec, tsize * sizeof(float4), cudaMemcpyDeviceToHost, s);
    cudaMemcpyAsync(hflags, flags, 2 * 4, cudaMemcpyDeviceToHost, s);
    cudaError_t e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) {
        cleanup();
        return cuda_err(c, e, "offset classes");
    }
    if (hflags[0]) {
        cleanup();
        return set_err(c, PD_ERR_UNSUPPORTED, "compact layout: a specimen with more offset classes than its table");
    }
    // templates, numbered per specimen in key order: a float vector xf and
    // the smallest bond length l0t of the class; |xf|^2, |xf|^2 - l0t^2 and
    // l0t as exact pairs
    std::vector<bt::Tpl> tp;
    std::vector<bt::Tpl3> tp3;
    std::vector<double> l0ts;
    std::vector<int> hid((size_t)tsize, -1), tbase((size_t)regions, 0);
    for (int64_t g = 0; g < regions; g++) {
        std::vector<std::pair<unsigned long long, int64_t>> used;
        for (int64_t h = 0; h < kRegion; h++)
            if (hk[g * kRegion + h] != kEmptyKey) used.push_back({hk[g * kRegion + h], g * kRegion + h});
        std::sort(used.begin(), used.end());
        if (used.size() > 255) {
            cleanup();
            return set_err(c, PD_ERR_UNSUPPORTED,
                           "compact layout: " + std::to_string(used.size()) + " offset classes in a specimen");
        }
        tbase[g] = (int)l0ts.size();
        for (size_t k = 0; k < used.size(); k++) {
            const unsigned long long key = used[k].first;
            const int64_t slot = used[k].second;
            hid[slot] = (int)k;
            float xf[3] = {0.0f, 0.0f, 0.0f};
            if (d3) {
                xf[0] = hv[slot].x, xf[1] = hv[slot].y, xf[2] = hv[slot].z;
            } else {
                xf[0] = bt::ffrom((uint32_t)(key >> 32)), xf[1] = bt::ffrom((uint32_t)key);
                // a component below 2^-74, whose scale is no float, counts as zero in
                // the template: offsets from zero are as exact (the key keeps it)
                for (int a = 0; a < 2; a++)
                    if (bt::class_scale(xf[a]) == 0.0f) xf[a] = 0.0f;
            }
            const int nd = d3 ? 3 : 2;
            double sh = 0.0, sl = 0.0;
            for (int a = 0; a < nd; a++) {
                const double sq = (double)xf[a] * (double)xf[a];  // exact: 24-bit significands
                const double t = sh + sq, bb = t - sh;
                sl += (sh - (t - bb)) + (sq - bb);
                sh = t;
            }
            const double l0t = bt::dfrom(hl[slot]);
            const double ph = l0t * l0t, pl = std::fma(l0t, l0t, -ph);
            const bt::f2 c0 = bt::split_bits((sh - ph) + (sl - pl));  // sh - ph exact (Sterbenz)
            const bt::f2 q0 = bt::split_bits(sh + sl);
            const bt::f2 l0 = bt::split_bits(l0t);
            l0ts.push_back(l0t);
            if (d3) {
                bt::Tpl3 T{};
                for (int a = 0; a < 3; a++) {
                    T.xf[a] = xf[a];
                    T.xd[a] = bt::dbits((double)xf[a]);
                    T.sc[a] = bt::class_scale(xf[a]);
                }
                T.c0h = c0.h, T.c0l = c0.l, T.q0h = q0.h, T.q0l = q0.l, T.l0h = l0.h, T.l0l = l0.l;
                T.l0d = l0t;
                tp3.push_back(T);
            } else {
                bt::Tpl T{};
                for (int a = 0; a < 2; a++) {
                    T.xf[a] = xf[a];
                    T.xd[a] = bt::dbits((double)xf[a]);
                }
                T.c0h = c0.h, T.c0l = c0.l, T.q0h = q0.h, T.q0l = q0.l, T.l0h = l0.h, T.l0l = l0.l;
                T.l0d = l0t;
                for (int a = 0; a < 2; a++) T.sc[a] = bt::class_scale(xf[a]);
                tp.push_back(T);
            }
        }
    }
    const size_t ntpl = l0ts.size();
    if (ntpl == 0) {
        cleanup();
        return set_err(c, PD_ERR_UNSUPPORTED, "compact layout: no bonds");
    }
    S.ntpl = (int)ntpl;
    const size_t nrec = (size_t)std::max<int64_t>(S.S, 1);
    bool ok = true;
    if (d3 && state)
        ok = mem.take(S.tpl3, ntpl * sizeof(bt::Tpl3)) && mem.take(S.srec8, nrec * sizeof(int2)) &&
             mem.take(S.stpl, ntpl * sizeof(StateTpl)) &&
             mem.take(S.bbits, (size_t)std::max<int64_t>(S.F, 1) * sizeof(uint32_t));
    else if (d3)
        ok = mem.take(S.tpl3, ntpl * sizeof(bt::Tpl3)) && mem.take(S.rec16, nrec * sizeof(bt::Rec));
    else if (state)
        ok = mem.take(S.tpl, ntpl * sizeof(bt::Tpl)) && mem.take(S.srec8, nrec * sizeof(int2)) &&
             mem.take(S.stpl, ntpl * sizeof(StateTpl));
    else
        ok = mem.take(S.tpl, ntpl * sizeof(bt::Tpl)) && mem.take(S.rec16, nrec * sizeof(bt::Rec));
    if (ok && regions > 1) ok = mem.take(S.inst_tbase, regions * sizeof(int));
    if (!ok) {
        cleanup();
        release();
        return set_err(c, PD_ERR_NOMEM, "compact records");
    }
    if (d3)
        cudaMemcpyAsync(S.tpl3, tp3.data(), ntpl * sizeof(bt::Tpl3), cudaMemcpyHostToDevice, s);
    else
        cudaMemcpyAsync(S.tpl, tp.data(), ntpl * sizeof(bt::Tpl), cudaMemcpyHostToDevice, s);
    cudaMemcpyAsync(ids, hid.data(), tsize * 4, cudaMemcpyHostToDevice, s);
    if (S.inst_tbase) cudaMemcpyAsync(S.inst_tbase, tbase.data(), regions * sizeof(int), cudaMemcpyHostToDevice, s);
    std::vector<StateTpl> st;
    if (state) {
        // logarithmic derivatives of the coefficients at each class's l0t: the
        // weight exp(-l0^2/delta^2) gives -2 l0 / delta^2; the partial-volume
        // factor (delta + dx/2 - l0) / dx (kernel_vol_Corr, Surf_Corr.cu:26-31)
        // above delta - dx/2 gives -1 / (delta + dx/2 - l0); l0 itself 1 / l0
        st.resize(ntpl);
        const double dlt = c->p.delta, hdx = c->p.dx / 2.0;
        for (size_t k = 0; k < ntpl; k++) {
            const double l0t = l0ts[k];
            double g2 = -2.0 * l0t / (dlt * dlt);
            if (l0t > dlt - hdx) g2 -= 1.0 / (dlt + hdx - l0t);
            st[k] = StateTpl{};
            st[k].g2 = (float)g2;
            st[k].g1 = (float)(g2 + 1.0 / l0t);
        }
        cudaMemcpyAsync(S.stpl, st.data(), ntpl * sizeof(StateTpl), cudaMemcpyHostToDevice, s);
    }
    if (d3 && !state) {
        k_rec16_fill3<<<dim3(gx, gy), 256, 0, s>>>(P, S.nslices, S.width, S.base, S.csr, c->NL, c->nf[PD_F_X],
                                                    c->nf[PD_F_Y], c->nf[PD_F_Z], c->idist, c->fac, c->scr, keys, ids,
                                                    S.tpl3, 0.5 * S.kscale_inv, S.rec16, flags + 1);
    } else if (d3) {
        k_state_compact3_fill<<<dim3(gx, gy), 256, 0, s>>>(
            P, S.nslices, S.width, S.base, S.csr, c->NL, c->nf[PD_F_X], c->nf[PD_F_Y], c->nf[PD_F_Z], c->idist, c->fac,
            c->w, keys, ids, S.tpl3, S.sn_exp, S.sth_exp, S.st_exp, S.srec8, S.stpl, flags + 1);
        k_break_bits<<<warps_grid(S.nslices), 256, 0, s>>>(P, S.nslices, S.width, S.base, S.fbase, S.csr,
                                                           c->nf[PD_F_Y], S.srec8, S.bbits);
        c->launches++;
    } else if (state) {
        k_state_compact_fill<<<dim3(gx, gy), 256, 0, s>>>(P, S.nslices, S.width, S.base, S.csr, c->NL, c->nf[PD_F_X],
                                                           c->nf[PD_F_Y], c->idist, c->fac, c->w, keys, ids, S.tpl,
                                                           S.sn_exp, S.sth_exp, S.st_exp, S.srec8, S.stpl,
                                                           flags + 1);
    } else {
        k_rec16_fill<<<warps_grid(S.nslices), 256, 0, s>>>(
            P, S.nslices, S.width, S.base, c->NN, c->rowptr, c->NL, grp, c->nf[PD_F_X], c->nf[PD_F_Y], c->idist, c->fac,
            c->scr, c->batch.node_bc, keys, ids, S.inst_tbase, S.tpl, -S.kexp, S.rec16, flags + 1);
    }
    c->launches++;
    if (state) {
        k_state_compact_check<<<dim3(gx, gy), 256, 0, s>>>(P, S.nslices, S.width, S.base, S.csr, c->idist, c->fac,
                                                            c->w, S.srec8, S.stpl, S.sn_exp, S.sth_exp, S.st_exp,
                                                            flags + 1);
        c->launches++;
    }
    cudaMemcpyAsync(hflags + 1, flags + 1, 4, cudaMemcpyDeviceToHost, s);
    e = cudaStreamSynchronize(s);
    cleanup();
    if (e != cudaSuccess) {
        release();
        return cuda_err(c, e, "compact records");
    }
    if (hflags[1]) {
        release();
        return set_err(c, PD_ERR_UNSUPPORTED, "compact layout: a bond outside its offset class's ranges");
    }
    return PD_OK;
}

int prepare(pd_ctx* c, cudaStream_t s) {
    if (!c->family) return set_err(c, PD_ERR_STATE, "prepare needs the bond family");
    drop_graphs(c);  // the SELL arrays are reallocated below
    DeviceBlocks& mem = c->blocks;
    const SetupCall call(mem, s, c->sell.width != nullptr);
    int rc;
    const bool state = c->p.model == PD_MODEL_STATE;
    if (state && !c->weights && (rc = initial_weight(c, s))) return rc;  // vol_corr included
    if (!c->volcorr && (rc = vol_corr(c, s))) return rc;
    // the SELL fail bits are rebuilt from the CSR flags
    if ((rc = sync_fail_to_csr(c, s))) return rc;
    const KParams P = kparams(c->p);
    Sell& S = c->sell;
    free_sell(c);
    S.nslices = (P.N + 31) / 32;
    cudaError_t e;
    if (!mem.take(S.width, S.nslices * sizeof(int)) || !mem.take(S.base, S.nslices * 8) ||
        !mem.take(S.fbase, (S.nslices + 1) * 8))
        return set_err(c, PD_ERR_NOMEM, "slice tables");
    k_slice_width<<<warps_grid(S.nslices), 256, 0, s>>>(P.N, S.nslices, c->NN, S.width);
    c->launches++;
    std::vector<int> w((size_t)S.nslices);
    if ((e = cudaMemcpyAsync(w.data(), S.width, w.size() * sizeof(int), cudaMemcpyDeviceToHost, s)) ||
        (e = cudaStreamSynchronize(s)))
        return cuda_err(c, e, "slice widths");
    std::vector<int64_t> fb((size_t)S.nslices + 1), bs((size_t)S.nslices);
    int64_t acc = 0;
    int wmax = 0;
    for (int64_t k = 0; k < S.nslices; k++) {
        fb[k] = acc;
        bs[k] = acc * 32;
        acc += w[k];
        wmax = std::max(wmax, w[k]);
    }
    fb[S.nslices] = acc;
    S.wmax = wmax;
    S.F = acc;
    S.S = acc * 32;
    cudaMemcpyAsync(S.fbase, fb.data(), fb.size() * 8, cudaMemcpyHostToDevice, s);
    cudaMemcpyAsync(S.base, bs.data(), bs.size() * 8, cudaMemcpyHostToDevice, s);
    const size_t n8 = (size_t)std::max<int64_t>(S.S, 1) * 8, n4 = (size_t)std::max<int64_t>(S.S, 1) * 4;
    bool ok = mem.take(S.csr, n4) && mem.take(S.bits, (size_t)std::max<int64_t>(S.F, 1) * 4);
    // every problem tries the compact layout first (small per-slot records on
    // offset-class templates); the 48-byte (bond-based) and three 32-byte
    // (state-based) records are the general layout, taken where the compact
    // one does not fit
    const bool try_compact = c->layout_pref != LAYOUT_RECORDS;
    if (ok && !state && !try_compact)
        ok = mem.take(S.rec, n8 * 6);
    // power-of-two scale bringing the bond coefficient 2 vol bc / dx near one,
    // so that the pair arithmetic of the force kernels stays in float range
    {
        const double ref = 2.0 * P.vol * P.bc / P.dx;
        S.kexp = (ref > 0.0 && std::isfinite(ref)) ? (int)std::lround(std::log2(ref)) : 0;
        S.kscale = std::ldexp(1.0, S.kexp);
        S.kscale_inv = std::ldexp(1.0, -S.kexp);
    }
    // state-based: powers of two near 1/m, the dilatation weight and the force
    // coefficient c2/m, from the lattice (m ~ half of delta^2 vol over a family
    // of pi (delta/dx)^2 or 4/3 pi (delta/dx)^3 members); any estimate within a
    // few binades keeps the pairs in float range, and the scalings are exact
    if (state) {
        const double r = P.delta / P.dx;
        const double nfam = P.dim == 2 ? M_PI * r * r : 4.0 / 3.0 * M_PI * r * r * r;
        const double m_est = 0.25 * P.delta * P.delta * P.vol * nfam;
        const double pr = P.pratio;
        const double th_coef = P.dim == 2 ? 2.0 * (2.0 * pr - 1.0) / (pr - 1.0) : 3.0;
        const double b_coef = P.dim == 2 ? 8.0 * P.G : 15.0 * P.G;
        auto lg = [](double v) { return (v > 0.0 && std::isfinite(v)) ? (int)std::lround(std::log2(v)) : 0; };
        S.sn_exp = lg(1.0 / m_est);
        S.sth_exp = -lg(std::fabs(th_coef) * P.delta * P.vol);
        S.st_exp = S.sn_exp + lg(std::fabs(2.0 * b_coef) * P.vol);
    }
    if (ok && state) ok = mem.take(S.e, n8) && !cudaMemsetAsync(S.e, 0, n8, s);
    if (ok && state && !try_compact)
        ok = mem.take(S.sgeo, n8 * 4) && mem.take(S.sth, n8 * 4) && mem.take(S.sfo, n8 * 4);
    if (!ok) {
        free_sell(c);
        return set_err(c, PD_ERR_NOMEM, "SELL bond arrays");
    }
    const unsigned gx = (unsigned)std::min<int64_t>(S.nslices, 65535);
    const unsigned gy = (unsigned)((S.nslices + gx - 1) / gx);
    k_sell_csr<<<warps_grid(S.nslices), 256, 0, s>>>(P.N, S.nslices, S.width, S.base, c->NN, c->rowptr, S.csr);
    c->launches++;
    if (!try_compact) {
        k_sell_fill<<<dim3(gx, gy), 256, 0, s>>>(P, S.nslices, S.width, S.base, c->NN, c->rowptr, c->NL, c->nf[PD_F_X],
                                                  c->nf[PD_F_Y], c->nf[PD_F_Z], c->idist, c->fac, c->scr, c->w,
                                                  c->nf[PD_F_M], c->batch.node_bc, c->batch.node_s0, S);
        c->launches++;
    } else {
        rc = build_compact(c, s);
        if (rc && c->layout_pref == LAYOUT_COMPACT) {
            free_sell(c);
            return rc;
        }
        if (rc) {
            // the general layout
            c->err.clear();
            if (state ? (!mem.take(S.sgeo, n8 * 4) || !mem.take(S.sth, n8 * 4) || !mem.take(S.sfo, n8 * 4))
                      : !mem.take(S.rec, n8 * 6)) {
                free_sell(c);
                return set_err(c, PD_ERR_NOMEM, "SELL bond arrays");
            }
            k_sell_fill<<<dim3(gx, gy), 256, 0, s>>>(P, S.nslices, S.width, S.base, c->NN, c->rowptr, c->NL,
                                                      c->nf[PD_F_X], c->nf[PD_F_Y], c->nf[PD_F_Z], c->idist, c->fac,
                                                      c->scr, c->w, c->nf[PD_F_M], c->batch.node_bc,
                                                      c->batch.node_s0, S);
            c->launches++;
        }
    }
    if (state) {
        k_inv_m<<<(unsigned)((P.N + 255) / 256), 256, 0, s>>>(P.N, c->nf[PD_F_M], std::ldexp(1.0, -S.sn_exp),
                                                             c->node_b, c->node_a);
        c->launches++;
    }
    c->bits_current = false;
    if ((rc = sync_fail_to_bits(c, s))) return rc;
    mem.trim();
    c->prepared = true;
    return cuda_err(c, cudaGetLastError(), "prepare");
}

}  // namespace pdg
