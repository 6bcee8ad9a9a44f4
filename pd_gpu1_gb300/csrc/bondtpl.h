// Per-bond arithmetic of the 2-D bond-based force kernels on lattice offset
// templates (the compact layout of force.cu: a 16-byte record per slot plus
// one template per lattice offset class).
//
// The reference computes, per bond (Force_Bond.cu:72-77),
//   d = ((x_c + u_c) - x_i) - u_i  (per component, FP64),
//   L = |d|, s = (L - l0) / l0,
//   f = vol fac bc scr s d / L,  broken when s > s0.
// Here d keeps the reference's FP64 roundings (P_c = x_c + u_c is stored per
// node, so d = (P_c - x_i) - u_i: two FP64 instructions per component; the 3-D
// and state-based kernels form it in one, see bond_squares in force.cu), and
// everything after d runs on pairs of floats (value h + l, about 48 bits):
//   eta = d - xf exactly, xf the offset class's float reference vector;
//   S   = eta . (2 xf + eta)  = |d|^2 - |xf|^2,
//   D   = S + c0 - 2 l0t dl   = L^2 - l0^2  (c0 = |xf|^2 - l0t^2, l0 = l0t + dl),
//   L^2 = S + |xf|^2,
//   e   = D / (L + l0)        = L - l0, without cancellation,
//   t   = (k2 / 2) e / L,  f += t (xf + eta)  with k2 = 2 vol fac bc scr / l0.
// Per bond that is four FP64 instructions (the reference's roundings of d) and
// about two hundred FP32 and integer instructions, against the reference's
// 58-odd FP64 instructions (three divides and a square root).
//
// The offset class (template) holds what every bond of one lattice offset
// shares: xf, |xf|^2, c0 and the class's reference length l0t (the smallest
// l0 of the class).  The slot keeps only what varies from row to row: the
// neighbour id, dl = l0 - l0t (a float: the bond lengths of one class differ
// in their last bits only), k2 and the class id (in the low byte of dl,
// whose significand has at most 15 bits).
//
// Plain C++ apart from the two approximate reciprocals, so that the host test
// suite compiles the same code and checks it against extended precision.
#pragma once
#include <math.h>
#include <stdint.h>
#include <string.h>

#include "exact_sub.h"

#if defined(__CUDACC__)
#define PD_BT_HD __host__ __device__ __forceinline__
#else
#define PD_BT_HD inline
#endif

namespace pdg {
namespace bt {

struct f2 {
    float h, l;  // value h + l
};

// One offset class: four 16-byte words, ordered so that a bond's stretch
// reads the first three (the fourth holds the scales of its offsets and l0t
// as a double, read only by the break test's exact path).
struct alignas(16) Tpl {
    uint64_t xd[2];  // xf as double bit patterns
    float xf[2];     // the class's float reference vector, components below 2^-74 as zero
    float c0h, q0h;  // c0 = |xf|^2 - l0t^2 and q0 = |xf|^2 as pairs (computed exactly),
    float c0l, q0l;  // their parts side by side for the packed sums
    float l0h, l0l;  // l0t as a pair
    float sc[2];     // ulp of xf as a double, with the sign of xf
    double l0d;      // l0t
};
static_assert(sizeof(Tpl) == 64, "four 16-byte words");

// One 3-D offset class: the same quantities as Tpl with three components
// (five 16-byte words; a stretch reads the first four).
struct alignas(16) Tpl3 {
    uint64_t xd[3];  // xf as double bit patterns
    float xf[3];     // the class's float reference vector
    float l0h;       // l0t as a pair, with l0l
    float c0h, q0h;  // c0 = |xf|^2 - l0t^2 and q0 = |xf|^2 as pairs, as in Tpl
    float c0l, q0l;
    float sc[3];     // ulp of xf as a double, with the sign of xf
    float l0l;
    double l0d;      // l0t
};
static_assert(sizeof(Tpl3) == 80, "five 16-byte words");

// Per-slot record: 16 bytes, one 128-bit load.
struct alignas(16) Rec {
    int col;      // neighbour id (the row itself for padding)
    float dl;     // l0 - l0t; the class id in the low 8 bits of its significand
    float k2h;    // k2 / 2 times 2^-kexp as a pair (zero for padding)
    float k2l;
};
static_assert(sizeof(Rec) == 16, "one 16-byte word");

PD_BT_HD uint32_t fbits(float f) {
#if defined(__CUDA_ARCH__)
    return __float_as_uint(f);
#else
    uint32_t u;
    memcpy(&u, &f, 4);
    return u;
#endif
}
PD_BT_HD float ffrom(uint32_t u) {
#if defined(__CUDA_ARCH__)
    return __uint_as_float(u);
#else
    float f;
    memcpy(&f, &u, 4);
    return f;
#endif
}
PD_BT_HD uint64_t dbits(double v) {
#if defined(__CUDA_ARCH__)
    return (uint64_t)__double_as_longlong(v);
#else
    uint64_t u;
    memcpy(&u, &v, 8);
    return u;
#endif
}
PD_BT_HD double dfrom(uint64_t u) {
#if defined(__CUDA_ARCH__)
    return __longlong_as_double((long long)u);
#else
    double v;
    memcpy(&v, &u, 8);
    return v;
#endif
}

// Error-free transformations (Knuth's TwoSum, Dekker's fast TwoSum for
// |a| >= |b| or a == 0, the FMA TwoProduct).
PD_BT_HD f2 two_sum(float a, float b) {
    const float s = a + b;
    const float bb = s - a;
    return f2{s, (a - (s - bb)) + (b - bb)};
}
PD_BT_HD f2 fast_sum(float a, float b) {
    const float s = a + b;
    return f2{s, b - (s - a)};
}
// The same operation on two floats, a bond's two components or its sums with c0
// and q0.  PK: one instruction for both (add, sub, mul and fma on an aligned pair
// of registers; each element rounds as the scalar operation does, so the results
// are the same bits, 53 instructions a 2-D bond fewer), where a kernel is short
// of issue slots; it takes a few more registers, and in a kernel that is short of
// those two instructions are faster (force.cu says which it is where).
template <bool PK>
struct v2 {
    float x, y;
};
#if defined(__CUDA_ARCH__)
#define PD_BT_V2(NAME)                                                                                             \
    __device__ __forceinline__ v2<true> v##NAME(v2<true> a, v2<true> b) {                                          \
        v2<true> r;                                                                                                \
        asm("{\n\t.reg .b64 a, b, c;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\t" #NAME                     \
            ".rn.f32x2 c, a, b;\n\tmov.b64 {%0, %1}, c;\n\t}"                                                      \
            : "=f"(r.x), "=f"(r.y)                                                                                 \
            : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));                                                             \
        return r;                                                                                                  \
    }                                                                                                              \
    __device__ __forceinline__ v2<false> v##NAME(v2<false> a, v2<false> b) {                                       \
        return v2<false>{__f##NAME##_rn(a.x, b.x), __f##NAME##_rn(a.y, b.y)};                                      \
    }
PD_BT_V2(add)
PD_BT_V2(sub)
PD_BT_V2(mul)
#undef PD_BT_V2
__device__ __forceinline__ v2<true> vfma(v2<true> a, v2<true> b, v2<true> c) {
    v2<true> r;
    asm("{\n\t.reg .b64 a, b, c, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmov.b64 c, {%6, %7};\n\t"
        "fma.rn.f32x2 d, a, b, c;\n\tmov.b64 {%0, %1}, d;\n\t}"
        : "=f"(r.x), "=f"(r.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return r;
}
__device__ __forceinline__ v2<false> vfma(v2<false> a, v2<false> b, v2<false> c) {
    return v2<false>{fmaf(a.x, b.x, c.x), fmaf(a.y, b.y, c.y)};
}
#else
template <bool PK>
inline v2<PK> vadd(v2<PK> a, v2<PK> b) { return v2<PK>{a.x + b.x, a.y + b.y}; }
template <bool PK>
inline v2<PK> vsub(v2<PK> a, v2<PK> b) { return v2<PK>{a.x - b.x, a.y - b.y}; }
template <bool PK>
inline v2<PK> vmul(v2<PK> a, v2<PK> b) { return v2<PK>{a.x * b.x, a.y * b.y}; }
template <bool PK>
inline v2<PK> vfma(v2<PK> a, v2<PK> b, v2<PK> c) { return v2<PK>{fmaf(a.x, b.x, c.x), fmaf(a.y, b.y, c.y)}; }
#endif
template <bool PK>
PD_BT_HD v2<PK> vneg(v2<PK> a) { return v2<PK>{-a.x, -a.y}; }

// Two pairs: value h + l per element.
template <bool PK>
struct p2 {
    v2<PK> h, l;
};
template <bool PK>
PD_BT_HD p2<PK> two_sum(v2<PK> a, v2<PK> b) {
    const v2<PK> s = vadd(a, b);
    const v2<PK> bb = vsub(s, a);
    return p2<PK>{s, vadd(vsub(a, vsub(s, bb)), vsub(b, bb))};
}
template <bool PK>
PD_BT_HD p2<PK> fast_sum(v2<PK> a, v2<PK> b) {
    const v2<PK> s = vadd(a, b);
    return p2<PK>{s, vsub(b, vsub(s, a))};
}

// a * b for pairs (relative error about 2^-47)
PD_BT_HD f2 mul(f2 a, f2 b) {
    const float p = a.h * b.h;
    float e = fmaf(a.h, b.h, -p);
    e = fmaf(a.h, b.l, e);
    e = fmaf(a.l, b.h, e);
    return fast_sum(p, e);
}

// FP32 estimates of 1/sqrt(x) and 1/x (the hardware's approximate
// instructions, relative error below 2^-22).  The host build, which has no
// such instructions, uses the correctly rounded values times a deterministic
// factor within 2^-22 of one, so that host checks of the refinements below
// see seeds as far off as the hardware's.
#if !defined(__CUDA_ARCH__)
PD_BT_HD float seed_noise(float x) {
    uint32_t h = fbits(x) * 2654435761u;
    h ^= h >> 15;
    return 1.0f + ldexpf((float)((int)(h & 0xffff) - 32768) / 32768.0f, -22);
}
#endif
PD_BT_HD float rsqrt_seed(float x) {
#if defined(__CUDA_ARCH__)
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
#else
    return (1.0f / sqrtf(x)) * seed_noise(x);
#endif
}
PD_BT_HD float rcp_seed(float x) {
#if defined(__CUDA_ARCH__)
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
#else
    return (1.0f / x) * seed_noise(x);
#endif
}

// 1/sqrt(x) of a positive pair from the FP32 estimate y0: with the residual
// rho = 1 - x y0^2 formed exactly enough (y0^2 and x.h y0^2 split by FMA),
// 1/sqrt(x) = y0 (1 - rho)^(-1/2) = y0 (1 + rho/2 + 3 rho^2/8 + ...); the
// second-order term leaves a relative error of about 3 rho^3 (below 1e-19),
// so the result is limited by the pair format alone.
PD_BT_HD f2 rsqrt2(f2 x) {
    const float y0 = rsqrt_seed(x.h);
    const float p = y0 * y0;
    const float pe = fmaf(y0, y0, -p);
    const float q = x.h * p;
    const float qe = fmaf(x.h, p, -q);
    const float c = fmaf(x.h, pe, fmaf(x.l, p, qe));
    const float rho = (1.0f - q) - c;
    return fast_sum(y0, y0 * fmaf(0.375f * rho, rho, 0.5f * rho));
}
// 1/z of a positive pair from the FP32 estimate r0: 1/z = r0 / (1 - rho) =
// r0 (1 + rho + rho^2 + ...), rho = 1 - z r0, to second order.
PD_BT_HD f2 rcp2(f2 z) {
    const float r0 = rcp_seed(z.h);
    const float q = z.h * r0;
    const float qe = fmaf(z.h, r0, -q);
    const float c = fmaf(z.l, r0, qe);
    const float rho = (1.0f - q) - c;
    return fast_sum(r0, r0 * fmaf(rho, rho, rho));
}

// diff * 2^(e - 1075) as a normalized pair with the sign of sgn (a float bit
// pattern whose sign bit is the value's), for |diff| < 2^48 and e in
// [949, 1120]: diff = hi 2^24 + lo with 0 <= lo < 2^24, both exact floats.
PD_BT_HD f2 pair_of_scaled(int64_t diff, int e, uint32_t sgn) {
    const float sc = ffrom((((uint32_t)(e - 948)) << 23) | (sgn & 0x80000000u));
    const float h = (float)(int)(diff >> 24) * (sc * 16777216.0f);
    const float l = (float)(int)(diff & 0xffffff) * sc;
    return fast_sum(h, l);
}

// eta = d - x exactly as a pair, x the double value of a float (xb its bit
// pattern).  Usual case: d and x of the same sign and binade, where the
// difference of the bit patterns is the difference of the significands; then
// operands within one binade of each other (sub_exact_scaled); otherwise the
// caller's fallback (returns false): split_bits(d) for x = 0, an FP64
// subtraction otherwise.
PD_BT_HD bool offset_pair(double d, uint64_t xb, f2& eta) {
    const uint64_t db = dbits(d);
    const uint32_t hd = (uint32_t)(db >> 32), hx = (uint32_t)(xb >> 32);
    const int eb = (int)((hd >> 20) & 0x7ffu);
    const int64_t df = (int64_t)(db - xb);
    if (((hd ^ hx) & 0xfff00000u) == 0 && (unsigned)(eb - 949) <= (unsigned)(1120 - 949) &&
        (uint64_t)(df + (1ll << 48)) < (uint64_t)(1ll << 49)) {
        eta = pair_of_scaled(df, eb, hd);
        return true;
    }
    int64_t diff;
    int e;
    if (sub_exact_scaled(db, xb, diff, e) && e >= 949 && e <= 1120 && diff < (1ll << 48) && diff > -(1ll << 48)) {
        eta = pair_of_scaled(diff, e, 0u);
        return true;
    }
    return false;
}

// ulp of a float's double, signed like it: the scale of offset_class (0 for
// zero).
PD_BT_HD float class_scale(float xf) {
    const uint32_t b = fbits(xf);
    const uint32_t E = (b >> 23) & 0xffu;
    return E < 53u ? 0.0f : ffrom((b & 0x80000000u) | ((E - 52u) << 23));
}

// offset_pair's usual case with the scale from the offset class: d and x of one
// sign and binade, whose exponent the class already knows (bit for bit
// offset_pair's result, in a third fewer instructions); false otherwise.
PD_BT_HD bool offset_class(double d, uint64_t xb, float sc, f2& eta) {
    const uint64_t db = dbits(d);
    const int64_t df = (int64_t)(db - xb);
    const float h = (float)(int)(df >> 24) * (sc * 16777216.0f);
    const float l = (float)(int)((uint32_t)df & 0xffffffu) * sc;
    eta = fast_sum(h, l);
    return (((uint32_t)(db >> 32) ^ (uint32_t)(xb >> 32)) & 0xfff00000u) == 0 &&
           (uint32_t)(df >> 32) + 0x10000u < 0x20000u;
}

// Double of a pair: fl(h + l) (both exact doubles).
PD_BT_HD double pair_sum_f64(f2 v) { return (double)v.h + (double)v.l; }

// A double as a pair with integer operations: h = v truncated to 24
// significant bits, l = the remaining 29 bits rounded to a float (relative
// error 2^-53; magnitudes below 2^-74 keep h only, below 2^-126 give zero).
PD_BT_HD f2 split_bits(double v) {
    const uint64_t b = dbits(v);
    const uint32_t hi = (uint32_t)(b >> 32), lo = (uint32_t)b;
    const uint32_t sign = hi & 0x80000000u, mag = hi & 0x7fffffffu;
    const uint32_t E = mag >> 20;
    const uint32_t hb = sign | ((mag - (896u << 20)) << 3) | (lo >> 29);
    const float rem = (float)(lo & 0x1fffffffu);
    const float scale = ffrom(((E - 948u) & 0xffu) << 23);  // 2^(E - 1075) when E >= 949
    const uint32_t lb = fbits(rem * scale) | sign;
    f2 r;
    r.h = E < 897u ? 0.0f : ffrom(hb);
    r.l = E < 949u ? 0.0f : ffrom(lb);
    return r;
}

struct BondOut {
    f2 f[2];  // force contribution per component, times 2^-kexp
    f2 e;     // extension L - l0
};

// D = S + c0 - 2 l0t dl = L^2 - l0^2 beside L^2 = S + |xf|^2, from S = eta . (2 xf
// + eta) in two parts.
template <bool PK, class TT>
PD_BT_HD void sums_with_class(float sh, float sl, const TT& T, float dl, f2& D, f2& L2) {
    p2<PK> d = two_sum(v2<PK>{sh, sh}, v2<PK>{T.c0h, T.q0h});
    d.l = vadd(vadd(v2<PK>{sl, sl}, d.l), v2<PK>{T.c0l, T.q0l});
    d.l.x = fmaf(-2.0f * T.l0h, dl, d.l.x);
    d = fast_sum(d.h, d.l);
    D = f2{d.h.x, d.l.x};
    L2 = f2{d.h.y, d.l.y};
}

// The stretch of one 2-D bond from its exact offsets eta (pairs), its
// offset class T and dl = l0 - l0t: the bond vector W = xf + eta, 1/L and the
// extension e = L - l0, all as pairs.
template <bool PK>
PD_BT_HD void stretch2(const p2<PK>& eta, const Tpl& T, float dl, p2<PK>& w, f2& y, f2& e) {
    // W = xf + eta and V = 2 xf + eta as pairs (TwoSum of the high parts)
    const v2<PK> xf{T.xf[0], T.xf[1]};
    w = two_sum(xf, eta.h);
    w.l = vadd(w.l, eta.l);
    p2<PK> v = two_sum(vadd(xf, xf), eta.h);  // 2 xf (exact)
    v.l = vadd(v.l, eta.l);
    // eta_a V_a: exact product of the high parts, cross terms in the low part
    const v2<PK> m = vmul(eta.h, v.h);
    v2<PK> lo = vfma(eta.h, v.h, vneg(m));
    lo = vfma(eta.h, v.l, lo);
    lo = vfma(eta.l, v.h, lo);
    // S = eta . V (the sum of the high parts exact; S_low carries the rest)
    const f2 s = two_sum(m.x, m.y);
    f2 D, L2;
    sums_with_class<PK>(s.h, (lo.x + lo.y) + s.l, T, dl, D, L2);
    // 1/L, L, L + l0, e = D / (L + l0)
    y = rsqrt2(L2);
    const f2 L = mul(L2, y);
    const f2 lp = two_sum(L.h, T.l0h);
    const f2 Lp = fast_sum(lp.h, ((lp.l + L.l) + T.l0l) + dl);
    e = mul(D, rcp2(Lp));
}

// A product of its own (no contraction into a sum).
PD_BT_HD float prod(float a, float b) {
#if defined(__CUDA_ARCH__)
    return __fmul_rn(a, b);
#else
    return a * b;
#endif
}

// ---- The stretch of the 3-D bond kernels and of the state-based passes ----
//
// The same quantities as stretch2 in fewer instructions, with an error no
// larger (tests/cpp/stretch_check.cpp holds both to quadruple precision): the
// bond vector W, D = L^2 - l0^2 and L^2 first (squares), then only what the
// pass needs, each from FP32 estimates and one Newton step whose residual is
// formed in pairs: the extension e (extension), e / L (stretch_ratio) or 1 / L
// (rsqrt2).  The 2-D bond-based kernels keep stretch2: the forces of a plate
// near rest are sums that cancel to a few of its last bits.

// W = xf + eta, D and L^2.  ORDERED: |eta_a.h| <= |xf_a|, or xf_a = 0, in
// every component, so that the two sums with eta may be fast ones.
template <int N, bool ORDERED, class TT>
PD_BT_HD void squares(const f2* eta, const TT& T, float dl, f2* w, f2& D, f2& L2) {
    // W = xf + eta, V = 2 xf + eta and eta V: x and y side by side
    const v2<true> xf{T.xf[0], T.xf[1]}, eh{eta[0].h, eta[1].h}, el{eta[0].l, eta[1].l};
    p2<true> q = ORDERED ? fast_sum(xf, eh) : two_sum(xf, eh);
    q.l = vadd(q.l, el);
    w[0] = f2{q.h.x, q.l.x}, w[1] = f2{q.h.y, q.l.y};
    const v2<true> x2 = vadd(xf, xf);
    p2<true> v = ORDERED ? fast_sum(x2, eh) : two_sum(x2, eh);
    v.l = vadd(v.l, el);
    // exact product of the high parts, cross terms in the low part
    const v2<true> m = vmul(eh, v.h);
    v2<true> r = vfma(eh, v.h, vneg(m));
    r = vfma(eh, v.l, r);
    r = vfma(el, v.h, r);
    f2 s = two_sum(m.x, m.y);
    float lows = s.l;
    s.l = r.x + r.y;
    if (N == 3) {  // z
        const f2 e3 = eta[N - 1];
        const float x3 = T.xf[N - 1], x32 = x3 + x3;
        const f2 q3 = ORDERED ? fast_sum(x3, e3.h) : two_sum(x3, e3.h);
        w[N - 1] = f2{q3.h, q3.l + e3.l};
        const f2 p3 = ORDERED ? fast_sum(x32, e3.h) : two_sum(x32, e3.h);
        const f2 v3{p3.h, p3.l + e3.l};
        const float m3 = prod(e3.h, v3.h);
        float r3 = fmaf(e3.h, v3.h, -m3);
        r3 = fmaf(e3.h, v3.l, r3);
        r3 = fmaf(e3.l, v3.h, r3);
        const f2 t = two_sum(s.h, m3);
        lows = lows + t.l;
        s = f2{t.h, s.l + r3};
    }
    sums_with_class<true>(s.h, s.l + lows, T, dl, D, L2);
}

// 1 / L within an ulp or two.
PD_BT_HD float rsqrt1(float x) {
    const float y0 = rsqrt_seed(x);
    return fmaf(0.5f * y0, fmaf(-prod(x, y0), y0, 1.0f), y0);
}

// a / b within an ulp or two.
PD_BT_HD float quotient1(float a, float b) {
    const float rb = rcp_seed(b);
    const float q = prod(a, rb);
    return fmaf(fmaf(-q, b, a), rb, q);
}

// e = L - l0 as the root of e (2 l0 + e) = D: no square root in pairs.
template <class TT>
PD_BT_HD f2 extension(f2 D, f2 L2, const TT& T, float dl) {
    const float y = rsqrt1(L2.h);
    const float e0 = quotient1(D.h, fmaf(L2.h, y, T.l0h));
    const f2 z = two_sum(T.l0h + T.l0h, e0);
    const float zl = z.l + 2.0f * (T.l0l + dl);
    const float p = prod(e0, z.h);
    const float pe = fmaf(e0, zl, fmaf(e0, z.h, -p));
    const float r = ((D.h - p) - pe) + D.l;  // D - e0 (2 l0 + e0); its slope is 2 L
    return fast_sum(e0, prod(r, 0.5f * y));
}

// g = e / L as the root of g (2 - g) L^2 = D; eh, e to FP32's precision.
template <class TT>
PD_BT_HD f2 stretch_ratio(f2 D, f2 L2, const TT& T, float& eh) {
    const float y = rsqrt1(L2.h);
    const float L = prod(L2.h, y);
    const float g0 = quotient1(D.h, fmaf(L, T.l0h, L2.h));
    eh = prod(g0, L);
    const float ah = 2.0f - g0, al = (2.0f - ah) - g0;
    const float ch = prod(ah, L2.h);
    const float ce = fmaf(al, L2.h, fmaf(ah, L2.l, fmaf(ah, L2.h, -ch)));
    const float p = prod(g0, ch);
    const float pe = fmaf(g0, ce, fmaf(g0, ch, -p));
    const float r = ((D.h - p) - pe) + D.l;  // D - g0 (2 - g0) L^2; its slope is 2 L l0
    return fast_sum(g0, prod(r, prod(y, 0.5f * rcp_seed(T.l0h))));
}

// The stretch of one 3-D bond whose vector is w = xf + eta: 1 / L and e.
PD_BT_HD void stretch3(const f2 eta[3], const Tpl3& T, float dl, f2 w[3], f2& y, f2& e) {
    f2 D, L2;
    squares<3, false>(eta, T, dl, w, D, L2);
    y = rsqrt2(L2);
    e = extension(D, L2, T, dl);
}

// The force contribution (times 2^-kexp) and the extension e of one 2-D bond.
template <bool PK>
PD_BT_HD p2<PK> bond2(const p2<PK>& eta, const Tpl& T, float dl, f2 k2half, f2& e) {
    p2<PK> w;
    f2 y;
    stretch2(eta, T, dl, w, y, e);
    // t = (k2 / 2) e / L, f = t W
    const f2 t = mul(mul(k2half, e), y);
    const v2<PK> th{t.h, t.h}, tl{t.l, t.l};
    const v2<PK> p = vmul(th, w.h);
    v2<PK> r = vfma(th, w.h, vneg(p));
    r = vfma(th, w.l, r);
    r = vfma(tl, w.h, r);
    return fast_sum(p, r);
}
PD_BT_HD BondOut bond2(const f2 eta[2], const Tpl& T, float dl, f2 k2half) {
    BondOut o;
    const p2<true> f = bond2(p2<true>{{eta[0].h, eta[1].h}, {eta[0].l, eta[1].l}}, T, dl, k2half, o.e);
    o.f[0] = f2{f.h.x, f.l.x};
    o.f[1] = f2{f.h.y, f.l.y};
    return o;
}

// a + b for pairs (TwoSum of the high parts, renormalized).
PD_BT_HD f2 add(f2 a, f2 b) {
    const f2 s = two_sum(a.h, b.h);
    return fast_sum(s.h, s.l + (a.l + b.l));
}

// Accumulate a pair into a running sum, renormalized at every addition (the
// low part stays within half an ulp of the high part, so the rounding of the
// low-part sum costs 2^-48 of the running sum, not of the low part's growth).
PD_BT_HD void acc_add(f2& acc, f2 v) {
    const f2 s = two_sum(acc.h, v.h);
    acc = fast_sum(s.h, s.l + (acc.l + v.l));
}

template <bool PK>
PD_BT_HD void acc_add(p2<PK>& acc, const p2<PK>& v) {
    const p2<PK> s = two_sum(acc.h, v.h);
    acc = fast_sum(s.h, vadd(s.l, vadd(acc.l, v.l)));
}

// acc + t w: as acc_add of the pair product, without renormalizing that.
PD_BT_HD void acc_prod(f2& acc, f2 t, f2 w) {
    const float p = prod(t.h, w.h);
    float e = fmaf(t.h, w.h, -p);
    e = fmaf(t.h, w.l, e);
    e = fmaf(t.l, w.h, e);
    const f2 s = two_sum(acc.h, p);
    acc = fast_sum(s.h, s.l + (acc.l + e));
}

PD_BT_HD void acc_prod(p2<true>& acc, f2 t, const f2* w) {
    const v2<true> wh{w[0].h, w[1].h}, wl{w[0].l, w[1].l}, th{t.h, t.h}, tl{t.l, t.l};
    const v2<true> p = vmul(th, wh);
    v2<true> e = vfma(th, wh, vneg(p));
    e = vfma(th, wl, e);
    e = vfma(tl, wh, e);
    const p2<true> s = two_sum(acc.h, p);
    acc = fast_sum(s.h, vadd(s.l, vadd(acc.l, e)));
}

// e > ecrit with ecrit = fl(s0 l0), l0 = l0t + dl, given s0 and s0f = s0
// rounded to float: decided on floats unless e lies within a few float ulps
// of the threshold (tf = s0f * l0h is within 4 ulps of ecrit), then on the
// double sum of the pair against the double threshold, the test of the
// reference-rounded kernels.
template <class TT>
PD_BT_HD bool exceeds(f2 e, double s0, float s0f, const TT& T, float dl) {
    const float tf = s0f * T.l0h;
    const int hb = (int)fbits(e.h), tb = (int)fbits(tf);
    if (hb >= tb + 8) return true;   // e >= e.h - ulp/2 > tf (1 + 2^-21) > ecrit
    if (hb < tb - 8) return false;   // e < tf (1 - 2^-21) < ecrit (e.h < 0 included)
    const double ecrit = s0 * (T.l0d + (double)dl);
    return pair_sum_f64(e) > ecrit;
}

// exceeds with an FP32 extension eh, within 2^-19 of e (relative, or of the
// threshold): where that does not decide, the pair does.
template <class TT>
PD_BT_HD bool exceeds_near(float eh, f2 D, f2 L2, double s0, float s0f, const TT& T, float dl) {
    const float tf = s0f * T.l0h;
    const int hb = (int)fbits(eh), tb = (int)fbits(tf);
    if (hb >= tb + 128) return true;
    if (hb < tb - 128) return false;
    return exceeds(extension(D, L2, T, dl), s0, s0f, T, dl);
}

// The exact double of a float from its IEEE fields (zero and subnormal
// floats give zero): no FP64 conversion instruction.
PD_BT_HD double f64_exact(float f) {
    const uint32_t b = fbits(f), mag = b & 0x7fffffffu;
    if (mag < 0x00800000u) return 0.0;
    const uint32_t hi = (b & 0x80000000u) | ((mag >> 3) + (896u << 20));
    return dfrom(((uint64_t)hi << 32) | (uint64_t)(uint32_t)(mag << 29));
}

// One component's term of the ADR damping numerator (kernel_cnn,
// Integrate.cu:17-33),
//   -u^2 (F/m - F_old/m) / (dt vh),
// as -u^2 ((F - F_old) (1/m)) / (dt vh) with both divisions through
// reciprocals: 1/m (IEEE-rounded, rmass) and 1/(dt vh) from the FP32
// estimate of the divisor's leading bits refined by two Newton steps in FP64
// (relative error near 2^-53).  About eleven FP64 instructions instead of the
// reference's two quotients and one IEEE division (about 24).  The term is
// within a few units in the last place of the exact value of the reference's
// formula (the reference's own evaluation loses more when F and F_old are
// close); the damping coefficient sums these terms over all nodes in another
// order than the reference's in any case.  Divisors outside [2^-100, 2^101)
// in magnitude take the IEEE division.
PD_BT_HD double damping_term(double u, double f, double fo, double rmass, double dt, double vh) {
    const double d = dt * vh;
    const double n = -1.0 * u * u * ((f - fo) * rmass);
    const uint64_t b = dbits(d);
    const uint32_t hi = (uint32_t)(b >> 32), lo = (uint32_t)b;
    const uint32_t mag = hi & 0x7fffffffu, E = mag >> 20;
    if (E < 923u || E > 1123u) return n / d;
    // d's leading bits as a float (truncated), then its reciprocal estimate
    const float df = ffrom((hi & 0x80000000u) | ((mag - (896u << 20)) << 3) | (lo >> 29));
    double y = f64_exact(rcp_seed(df));
    y = fma(y, fma(-d, y, 1.0), y);
    y = fma(y, fma(-d, y, 1.0), y);
#if defined(__CUDA_ARCH__)
    return __dmul_rn(n, y);  // a product of its own (no contraction into the caller's sum)
#else
    return n * y;
#endif
}

}  // namespace bt
}  // namespace pdg
