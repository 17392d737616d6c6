// gd_fixed.cuh -- scaled 64-bit integer arithmetic for the step's face solvers.
//
// GB300's FP64 unit takes 64 cycles of an SM sub-partition per warp instruction, the integer
// pipes two for an add or a shift and four for a 32x32->64 multiply-add (measured: 1.88 DFMA,
// 59 64-bit adds, 25 wide multiply-adds per clock and SM; all three run side by side).  A face
// flux is a short chain of products and sums of quantities of a few known sizes, so it can be
// formed in integers: each quantity is a signed 64-bit integer times a power of two chosen per
// face from the exponents of its cells (one per state component, one for the face's normal
// velocities and speeds, ...).  A sum is then one 64-bit add, a product mulk() below, and nothing
// is rounded to 53 bits before the result is.
//
// Host-compilable, so that the same arithmetic is checked on the CPU against 113-bit floats.
#pragma once

#include <cmath>
#include <cstdint>

#include "gd_swfp.cuh"

namespace gd {
namespace fx {

using i64 = long long;
using u64 = unsigned long long;

GD_HD int32_t hi32(i64 x) { return (int32_t)(x >> 32); }
GD_HD uint32_t lo32(i64 x) { return (uint32_t)x; }

// x y / 2^(64 - KX - KY), |x| < 2^(63 - KX), |y| < 2^(63 - KY), to 3 units below (ROUND: the
// dropped bits' mean is added, 0 stays 0).  Three wide multiply-adds: the product of the low
// words and their lowest bits are left out.  Inline PTX: from the same C++ the compiler makes
// twice the instructions (63 against 26 for four products, ncu).
template <int KX, int KY, bool ROUND = true>
GD_HD i64 mulk(i64 x, i64 y) {
    x = (i64)((u64)x << KX);
    y = (i64)((u64)y << KY);
#if defined(__CUDA_ARCH__)
    i64 r;
    asm("{\n\t.reg .s32 xl, xh, yl, yh;\n\t.reg .s64 c;\n\t"
        "mov.b64 {xl, xh}, %1;\n\t"
        "mov.b64 {yl, yh}, %2;\n\t"
        "shr.u32 xl, xl, 1;\n\t"
        "shr.u32 yl, yl, 1;\n\t"
        "mad.wide.s32 c, xh, yl, %3;\n\t"
        "mad.wide.s32 c, yh, xl, c;\n\t"
        "shr.s64 c, c, 31;\n\t"
        "mad.wide.s32 %0, xh, yh, c;\n\t}"
        : "=l"(r) : "l"(x), "l"(y), "n"(ROUND ? 0x7fffffff : 0));
    return r;
#else
    const int32_t xh = hi32(x), yh = hi32(y);
    const int32_t xl = (int32_t)(lo32(x) >> 1), yl = (int32_t)(lo32(y) >> 1);
    return (i64)xh * yh +
           (((i64)xh * yl + ((i64)yh * xl + (ROUND ? 0x7fffffffLL : 0LL))) >> 31);
#endif
}
// x y / 2^32 for 0 <= y < 2^31
GD_HD i64 mul32(i64 x, uint32_t y) {
#if defined(__CUDA_ARCH__)
    i64 r;
    asm("{\n\t.reg .b32 xl, xh, t;\n\t.reg .b64 c;\n\t"
        "mov.b64 {xl, xh}, %1;\n\t"
        "mul.hi.u32 t, xl, %2;\n\t"
        "mov.b64 c, {t, 0};\n\t"
        "mad.wide.s32 %0, xh, %2, c;\n\t}"
        : "=l"(r) : "l"(x), "r"(y));
    return r;
#else
    return (i64)((u64)((i64)hi32(x) * (i64)(int32_t)y) + (((u64)lo32(x) * y) >> 32));
#endif
}
GD_HD u64 umul32(u64 x, uint32_t y) {  // the same for x up to 2^64
#if defined(__CUDA_ARCH__)
    u64 r;
    asm("{\n\t.reg .b32 xl, xh, t;\n\t.reg .b64 c;\n\t"
        "mov.b64 {xl, xh}, %1;\n\t"
        "mul.hi.u32 t, xl, %2;\n\t"
        "mov.b64 c, {t, 0};\n\t"
        "mad.wide.u32 %0, xh, %2, c;\n\t}"
        : "=l"(r) : "l"(x), "r"(y));
    return r;
#else
    return (u64)(uint32_t)(x >> 32) * y + (((u64)(uint32_t)x * y) >> 32);
#endif
}
GD_HD i64 wide(int32_t x, int32_t y) {  // x y
#if defined(__CUDA_ARCH__)
    i64 r;
    asm("mul.wide.s32 %0, %1, %2;" : "=l"(r) : "r"(x), "r"(y));
    return r;
#else
    return (i64)x * y;
#endif
}

GD_HD int clz32(uint32_t x) {  // 32 for 0
#if defined(__CUDA_ARCH__)
    return __clz((int)x);
#else
    return x ? __builtin_clz(x) : 32;
#endif
}
GD_HD int clz64(u64 x) {  // 64 for 0
#if defined(__CUDA_ARCH__)
    return __clzll((i64)x);
#else
    return x ? __builtin_clzll(x) : 64;
#endif
}
GD_HD int imax(int a, int b) { return a > b ? a : b; }
GD_HD int imin(int a, int b) { return a < b ? a : b; }
// arithmetic shift right by any n >= 0
GD_HD i64 sra(i64 x, int n) { return x >> (n < 63 ? n : 63); }

// x 2^-s for either sign of s; a left shift's result fits
GD_HD i64 shift(i64 x, int s) {
    return (i64)((u64)x << imin(imax(-s, 0), 62)) >> imin(imax(s, 0), 63);
}
GD_HD i64 iabs(i64 x) { return x < 0 ? -x : x; }
// whether x >= 0 shifted by shift(x, s) stays below 2^61
GD_HD bool fits(i64 x, int s) { return s >= 0 || x >> imax(61 + s, 0) == 0; }

GD_HD float rsqrt_seed(float x) {
#if defined(__CUDA_ARCH__)
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
#else
    return 1.0f / std::sqrt(x);
#endif
}
GD_HD float rcp_seed(float x) {
#if defined(__CUDA_ARCH__)
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
#else
    return 1.0f / x;
#endif
}

// A positive normal double as m 2^(e - 62), m in [2^62, 2^63); e is its unbiased exponent.
struct Pos {
    i64 m;
    int e;
};
GD_HD Pos pos_of(double x) {
    uint32_t hi, lo;
    swfp::halves(x, hi, lo);
    Pos p;
    p.e = (int)(hi >> 20) - 1023;
    const uint32_t h = (hi & 0xfffffu) | 0x100000u;
    p.m = (i64)(((u64)((h << 10) | (lo >> 22)) << 32) | (lo << 10));
    return p;
}
// a signed state in units of 2^(top - 61) as m 2^(e - 62), m as large as fits unless tiny
GD_HD Pos signed_of(i64 a, int top) {
    const int32_t h = hi32(a);
    const int z = clz32((uint32_t)(h ^ (h >> 31))) - 1;
    return Pos{a << z, top + 1 - z};
}

// 1 / x for x > 0 with a nonzero high word: r 2^(lz - 124), lz the leading zeros of x, r in
// (2^60, 2^61).  The FP32 reciprocal y of the leading 24 bits, then y (1 + e + e^2) with
// e = 1 - x y (Newton's iteration with the quadratic term kept) in units of 2^-62.
GD_HD i64 rcp(i64 x, int& lz) {
    lz = clz32((uint32_t)hi32(x));
    const u64 n = (u64)x << lz;
    const float f = swfp::f32_from_bits(0x3f800000u | ((uint32_t)(n >> 40) & 0x7fffffu));
    // y in [1/2, 1] as an integer of unit 2^-31 (the pattern's step at 1 keeps this linear)
    const uint32_t y = ((swfp::bits_of_f32(rcp_seed(f)) - 0x3e800000u) << 7) - 1u;
    const i64 e = (i64)(0x4000000000000000ULL - umul32(n, y));
    const int32_t es = (int32_t)(e >> 20);
    const i64 g = e + (wide(es, es) >> 22);
    return ((i64)((u64)y << 30) - 1) + mul32(g, y);
}

// sqrt(a / r) of a = am 2^(ea - 60), am in [2^60, 2^62), and r = rm 2^(er - 62): w 2^(k - 60),
// w in [2^58, 2^61).  The FP32 seed y of 1/sqrt(a r), w = a y, e = 1 - w (r y), and
// w (1 + e/2 + 3 e^2 / 8), the series of 1/sqrt(1 - e).
GD_HD i64 sqrt_over(i64 am, int ea, Pos r, int& k) {
    const int d = ea - r.e + 2;
    k = d >> 1;
    const i64 a = am << (d & 1);
    const float f = (float)hi32(a) * (float)hi32(r.m);
    // 2^60 y, between 2^29 and 2^31
    const uint32_t y = (uint32_t)(rsqrt_seed(f) * 1152921229728940032.0f);
    const i64 w = mul32(a, y), t = mul32(r.m, y);
    const i64 e = (1LL << 59) - mulk<2, 1, false>(w, t);
    const int32_t es = (int32_t)(e >> 16);
    const i64 g = (e << 2) + (wide(es, 3 * es) >> 27);
    return w + (mulk<0, 0, false>(w, g << 21) >> 19);
}

// The constants a face solver needs of gamma, as m 2^(e - 62).
struct Gas {
    i64 g, gg, gi;  // gamma, gamma / (gamma - 1), 1 / (gamma - 1)
    int ge, gge, gie;
    int room;     // extra bits that gamma / (gamma - 1) p takes beside rho c^2; -1: no integer path
};
inline Gas gas_of(double gamma) {
    Gas G;
    const Pos a = pos_of(gamma), b = pos_of(gamma / (gamma - 1.0)), c = pos_of(1.0 / (gamma - 1.0));
    G.gi = c.m;
    G.gie = c.e;
    G.g = a.m;
    G.ge = a.e;
    G.gg = b.m;
    G.gge = b.e;
    G.room = b.e > 2 ? b.e - 2 : 0;
    if (a.e > 16 || b.e > 16) G.room = -1;  // gamma beyond 2^16, or within 2^-16 of 1
    return G;
}

// 0 unless a and b have the same sign, else the one of smaller magnitude
GD_HD i64 minmod(i64 a, i64 b) {
    const bool lt = a < b, neg = hi32(a) < 0;
    const i64 m = lt != neg ? a : b;
    return (hi32(a) ^ hi32(b)) < 0 ? 0 : m;
}

GD_HD uint32_t rotate(uint32_t x, int n) {  // by 0 or 16 bits
#if defined(__CUDA_ARCH__)
    return __funnelshift_l(x, x, n);
#else
    return n ? x << 16 | x >> 16 : x;
#endif
}

// ---- cells and the states of a face ------------------------------------------------------------
//
// A cell is held as the signed significands of its values, x = q 2^(e - 60) with q below 2^61, and
// the exponent fields e, packed 16 bits each (Keys).  A face takes, per component, the unit
// 2^(top - 60) from the cells of its own stencil, so that a shift is all that separates a cell from
// the face's integers: what a face computes depends on its stencil alone, and a small component
// beside large ones, or a quiet cell in a tile with a shock, keeps its digits.
constexpr int kSpan = 8;     // exponents that the face's densities, and the pressures, may span
constexpr int kRange = 128;  // exponents of densities, pressures (both signs) and velocities
constexpr uint32_t kNoKey = 0x7ff;  // key of a value that the integers do not take

// {rho, p}, {vx, vy}, {bx, by}, {bz, 0}
template <int NF>
struct alignas(NF == 4 ? 8 : 16) Keys {
    static constexpr int W = NF == 4 ? 2 : 4;
    uint32_t w[W];
};
// the larger and the smaller of both 16-bit halves
GD_HD uint32_t max2(uint32_t a, uint32_t b) {
#if defined(__CUDA_ARCH__)
    return __vmaxu2(a, b);
#else
    const uint32_t l = (a & 0xffffu) > (b & 0xffffu) ? a : b, h = (a >> 16) > (b >> 16) ? a : b;
    return (l & 0xffffu) | (h & 0xffff0000u);
#endif
}
GD_HD uint32_t min2(uint32_t a, uint32_t b) {
#if defined(__CUDA_ARCH__)
    return __vminu2(a, b);
#else
    const uint32_t l = (a & 0xffffu) < (b & 0xffffu) ? a : b, h = (a >> 16) < (b >> 16) ? a : b;
    return (l & 0xffffu) | (h & 0xffff0000u);
#endif
}
// x / 2^n below, n any number that is not negative
GD_HD i64 asr(i64 x, uint32_t n) {
#if defined(__CUDA_ARCH__)
    i64 r;
    asm("shr.s64 %0, %1, %2;" : "=l"(r) : "l"(x), "r"(n));  // amounts beyond 63 act as 63
    return r;
#else
    return x >> (n < 63 ? n : 63);
#endif
}
// The significand and the key of a cell's value: a density or pressure (POSITIVE), or a component
// of a vector.
template <bool POSITIVE>
GD_HD uint32_t cell_units(double x, i64& q) {
    uint32_t hi, lo;
    swfp::halves(x, hi, lo);
    const uint32_t e = (hi >> 20) & 0x7ffu;
    const uint32_t h = (hi & 0xfffffu) | (e ? 0x100000u : 0u);
    const i64 m = (i64)(((u64)((h << 8) | (lo >> 24)) << 32) | (lo << 8));
    q = (int32_t)hi < 0 ? -m : m;
    if (POSITIVE) return (hi >> 20) - 1u < 0x7feu ? e : kNoKey;  // zeros and negatives out
    return e != 0 || m == 0 ? e : kNoKey;  // subnormal numbers out
}
template <int NF>
GD_HD void cell_units(const double* v, i64* q, int fs, Keys<NF>& k) {
    uint32_t e[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
    for (int f = 0; f < NF; ++f)
        e[f] = f < 2 ? cell_units<true>(v[f], q[f * fs]) : cell_units<false>(v[f], q[f * fs]);
#pragma unroll
    for (int w = 0; w < Keys<NF>::W; ++w) k.w[w] = e[2 * w] | (e[2 * w + 1] << 16);
}
// the field of the local frame's component f: x-face (n, t) = (x, y); y-face (n, t) = (y, x)
GD_HD int face_field(int f, bool isx) {
    return isx || f < 2 || f == 6 ? f : (f < 4 ? 5 - f : 9 - f);
}

// c + d/2 and c - d/2 of the cells on either side of a face, d the minmod slopes (ORDER 1: c), per
// component of the face's local frame in units of 2^(top - 61), below 2^62.  q, key: the cell above
// the face; its neighbours along the normal are st (in key: kst) apart, its fields fs.  False where
// a cell of the stencil is out of the integers' range.
//
// The unit is that of the two cells beside the face, up to 3 exponents above them if the outer
// cells are larger.  An outer cell beyond that stays as it is, at 8 times the inner cells' exponent
// or above: its difference keeps the sign and stays the larger one, which is all minmod asks of it.
template <int NF, int ORDER>
GD_HD bool face_states(const i64* q, int st, int fs, const Keys<NF>* key, int kst, bool isx, i64* a,
                       i64* b, int* top) {
    constexpr int W = Keys<NF>::W;
    const Keys<NF> ka = key[-kst], kb = key[0];
    Keys<NF> k1, k2, kt;  // the outer cells, the units
    uint32_t high = 0;
#pragma unroll
    for (int w = 0; w < W; ++w) {
        const uint32_t m = max2(ka.w[w], kb.w[w]);
        kt.w[w] = m;
        if (ORDER == 2) {
            k1.w[w] = key[-2 * kst].w[w];
            k2.w[w] = key[kst].w[w];
            const uint32_t o = max2(k1.w[w], k2.w[w]);
            high = max2(high, o);
            kt.w[w] = max2(m, min2(o, m + 0x30003u));
        }
        high = max2(high, m);
    }
    const uint32_t low = min2(ka.w[0], kb.w[0]);
    constexpr uint32_t kH = (1023 + kRange) * 0x10001u, kL = (1023 - kRange) * 0x10001u;
    constexpr uint32_t kS = kSpan * 0x10001u;
    if (max2(high, kH) != kH || min2(low, kL) != kL || max2(kt.w[0] - low, kS) != kS) return false;
    // shifts, and the units, in the local frame
    uint32_t sa[W], sb[W], s1[W], s2[W];
#pragma unroll
    for (int w = 0; w < W; ++w) {
        uint32_t t = kt.w[w];
        sa[w] = t - ka.w[w];
        sb[w] = t - kb.w[w];
        if (ORDER == 2) {
            s1[w] = t - min2(k1.w[w], t);
            s2[w] = t - min2(k2.w[w], t);
        }
        if (w == 1 || w == 2) {
            const int r = isx ? 0 : 16;
            t = rotate(t, r);
            sa[w] = rotate(sa[w], r);
            sb[w] = rotate(sb[w], r);
            if (ORDER == 2) {
                s1[w] = rotate(s1[w], r);
                s2[w] = rotate(s2[w], r);
            }
        }
        kt.w[w] = t;
    }
#pragma unroll
    for (int f = 0; f < NF; ++f) {
        const int w = f >> 1, h = 16 * (f & 1);
        const i64* p = q + face_field(f, isx) * fs;
        const i64 ca = asr(p[-st], sa[w] >> h & 0xffffu), cb = asr(p[0], sb[w] >> h & 0xffffu);
        a[f] = 2 * ca;
        b[f] = 2 * cb;
        if (ORDER == 2) {  // between the cell and the middle to its neighbour: rho, p > 0
            const i64 d = cb - ca;
            a[f] += minmod(ca - asr(p[-2 * st], s1[w] >> h & 0xffffu), d);
            b[f] -= minmod(d, asr(p[st], s2[w] >> h & 0xffffu) - cb);
        }
        top[f] = (int)(kt.w[w] >> h & 0xffffu) - 1023;
    }
    return true;
}

// x 2^ue as a double, a normal number or 0: ue is added to the exponent field.  Densities, pressures
// and fan speeds of the accepted range make normal numbers of every flux but those that a tangential
// velocity or a field enters alone: for them the sign bit of `bad` is set where the result is no
// normal number, and the face goes to the floating-point solver.
GD_HD double to_double(i64 x, int ue) {
    uint32_t hi, lo;
    swfp::halves((double)x, hi, lo);  // hi is 0 for x = 0 alone
    return swfp::from_halves(hi + (hi == 0 ? 0u : (uint32_t)ue << 20), lo);
}
GD_HD double to_double(i64 x, int ue, uint32_t& bad) {
    uint32_t hi, lo;
    swfp::halves((double)x, hi, lo);
    const uint32_t r = hi + (hi == 0 ? 0u : (uint32_t)ue << 20);
    bad |= (r - (hi == 0 ? 0u : 0x100000u)) ^ hi;
    return swfp::from_halves(r, lo);
}
// E for which both x 2^(top - 61) and y 2^(top - 61) are below 2^(E - 1), from their leading words:
// the least one, and at least top - 28
GD_HD int top_of(i64 x, i64 y, int top) {
    const int32_t h = hi32(x), k = hi32(y);
    return top + 4 - clz32((uint32_t)((h ^ (h >> 31)) | (k ^ (k >> 31))));
}
// at least top
GD_HD int scale_of(i64 x, i64 y, int top) { return imax(top_of(x, y, top), top); }

// The two sides of a face in its local frame, per component (rho, p, normal and tangential
// velocity) in units of 2^(X - 61), below 2^62.
struct Tops {
    int r, p, n, t;
};
struct States {
    i64 rL, rR, pL, pR, uL, uR, vL, vR;
};
// a positive state in units of 2^(top - 61), its high word not 0
GD_HD Pos pos_of(i64 a, int top) {
    const int lz = clz32((uint32_t)hi32(a));
    return Pos{a << (lz - 1), top - lz + 2};
}

// The wave speeds of a face, all velocities in units of 2^(E - 61).  |u|, c < 2^(E - 1), so
// |S| < 2^61 and |S - u| < 1.5 2^61 in these units.
struct Fan {
    Pos RL, RR, PL, PR;
    i64 uL, uR, SL, SR;
    int E, kmin;  // kmin: 2^kmin is about the smaller sound speed
    bool ok;
};
// ok is false where a scale would leave a quantity fewer bits than binary64 does: accepted are
// sound speeds within a factor of about 4 of each other, and normal velocities to about 2^22 of
// them (the larger velocity is then the scale of every flux).  UU: the larger wave speed.
// HLL: the fan min(u) - max(c), max(u) + max(c) of kernel.cu:1516-1517 instead of Davis'.
template <bool HLL = false>
GD_HD Fan fan_of(const States& q, const Tops& X, const Gas& G, double& UU) {
    Fan f;
    f.RL = pos_of(q.rL, X.r);
    f.RR = pos_of(q.rR, X.r);
    f.PL = pos_of(q.pL, X.p);
    f.PR = pos_of(q.pR, X.p);
    int kL, kR;
    const i64 wL = sqrt_over(mulk<0, 0>(f.PL.m, G.g), f.PL.e + G.ge, f.RL, kL);
    const i64 wR = sqrt_over(mulk<0, 0>(f.PR.m, G.g), f.PR.e + G.ge, f.RR, kR);
    const int kmax = imax(kL, kR);
    f.kmin = imin(kL, kR);
    f.E = imax(kmax + 2, scale_of(q.uL, q.uR, X.n));
    f.ok = kmax - f.kmin <= 2 && f.E - kmax <= 24;
    if (!f.ok) return f;
    i64 cL = wL >> (f.E - 1 - kL), cR = wR >> (f.E - 1 - kR);
    if (HLL) {
        cL = cL > cR ? cL : cR;
        cR = cL;
    }
    const int sh = imin(f.E - X.n, 63);
    f.uL = q.uL >> sh;
    f.uR = q.uR >> sh;
    const i64 aL = f.uL - cL, aR = f.uR - cR, bL = f.uL + cL, bR = f.uR + cR;
    f.SL = aL < aR ? aL : aR;
    f.SR = bL > bR ? bL : bR;
    UU = to_double(-f.SL > f.SR ? -f.SL : f.SR, f.E - 61);
    return f;
}

// HLLC flux (mass, normal and tangential momentum, energy) of that face: the formulas of
// hllc_local.  Returns false, with nothing formed, where the face lies inside the fan and a
// velocity is more than about 4 sound speeds; the caller then takes hllc_local.  SL < S_M < SR
// (the Davis speeds, with positive pressures), and inside the fan S_M and S have opposite signs,
// so |S_M / (S - S_M)| <= 1: no product below overflows.
GD_HD bool hllc(const Fan& f, const States& s, const Tops& X, const Gas& G, double& Fm,
                double& Fn, double& Ft, double& Fe) {
    uint32_t bad = 0;
    const int E = f.E, ER = imax(f.RL.e, f.RR.e);
    const i64 suL = f.SL - f.uL, suR = f.SR - f.uR;
    // r (S - u), each side in units of its own density's, 2^(e + E - 59), and in the larger's
    const i64 oL = mulk<0, 0>(f.RL.m, suL), oR = mulk<0, 0>(f.RR.m, suR);
    const i64 mL = oL >> (ER - f.RL.e), mR = oR >> (ER - f.RR.e);
    const i64 D = mR - mL;
    // units 2^(ER + 2E - 60)
    const int sp = ER + 2 * E + 2;
    const i64 N = mulk<1, 3>(mR, f.uR) - mulk<1, 3>(mL, f.uL) +
                  ((f.PL.m >> imin(sp - f.PL.e, 63)) - (f.PR.m >> imin(sp - f.PR.e, 63)));
    int lz;
    const i64 iD = rcp(D, lz);
    i64 SM = mulk<0, 2>(N << (lz - 2), iD);

    const bool takeL = f.SL > 0 || N >= 0;
    const bool star = takeL ? f.SL <= 0 : f.SR >= 0;
    const Pos R{takeL ? f.RL.m : f.RR.m, takeL ? f.RL.e : f.RR.e};
    const Pos Pk{takeL ? f.PL.m : f.PR.m, takeL ? f.PL.e : f.PR.e};
    const i64 un = takeL ? f.uL : f.uR, S = takeL ? f.SL : f.SR;
    const i64 o = takeL ? oL : oR;
    const Pos T = signed_of(takeL ? s.vL : s.vR, X.t);

    i64 qs = un;  // outside the fan the physical flux: S_M -> u, q (S - u) -> u
    if (star) {
        if (E - f.kmin > 3) return false;
        const i64 su = takeL ? suL : suR;
        const i64 ad = takeL ? SM - S : S - SM;
        if (hi32(ad) <= 0) return false;
        int lz2;
        const i64 iA = rcp(ad, lz2);
        const i64 q = mulk<0, 2>(SM << (lz2 - 2), iA);  // |S_M / (S - S_M)| 2^60, signed as S_M
        qs = mulk<2, 1>(takeL ? -q : q, su) << 1;
    } else {
        SM = un;
    }
    const i64 SMu = SM - un;
    const int32_t qh = hi32(qs);
    const int z = clz32((uint32_t)(qh ^ (qh >> 31))) - 1;
    const i64 qn = qs << z;
    const i64 M = mulk<0, 0>(R.m, qn);
    const int em = R.e + E - 59 - z;
    Fm = to_double(M, em);
    // momentum: p + r q su S_M + r su (S_M - u); exactly p where the rest is 0
    const i64 t = (mulk<1, 2>(M, SM) >> z) + mulk<2, 1>(o, SMu);
    const int et = R.e + 2 * E - 59;
    const i64 pt = (Pk.m >> imin(et - Pk.e + 62, 63)) + t;
    Fn = to_double(t == 0 ? Pk.m : pt, t == 0 ? Pk.e - 62 : et);
    const i64 MT = mulk<0, 0>(M, T.m);
    Ft = to_double(MT, em + T.e + 2, bad);
    // energy: q su (p gamma / (gamma - 1) + r (u^2 / 2 + S (S_M - u))) + (mass flux) v^2 / 2
    const i64 H = mulk<1, 1>(un, un) + mulk<2, 1>(S, SMu);
    const i64 B = sra(mulk<0, 0>(Pk.m, G.gg), R.e + 2 * E - Pk.e - G.gge + G.room) +
                  (mulk<0, 1>(R.m, H) >> G.room);
    const i64 e1 = mulk<0, 0>(qn, B);
    const i64 e2 = mulk<2, 0>(MT, T.m);
    const int dx = 2 * (E - T.e) + 1 + G.room;
    const int x1 = R.e + 3 * E - 57 - z + G.room;
    Fe = to_double(sra(e1, imax(-dx, 0)) + sra(e2, imax(dx, 0)), dx > 0 ? x1 : x1 - dx);
    return (int32_t)bad >= 0;
}

// HLL flux of that face (kernel.cu:1485-1609) with fan_of<true>.  With the fan cut at the face,
// D_L <= 0 <= D_R, and a = D_R / (D_R - D_L), the average (D_R F_L - D_L F_R + D_L D_R (U_R - U_L))
// / (D_R - D_L) is a (F_L - D_L U_L) + (1 - a) (F_R - D_R U_R), and on one side of the face
// a = 1 or 0 gives the physical flux: no difference of the two sides' states is formed.  False,
// with nothing to use, where the energy would not fit its unit.
GD_HD bool hll(const Fan& f, const States& s, const Tops& X, const Gas& G, double& Fm, double& Fn,
               double& Ft, double& Fe) {
    uint32_t bad = 0;
    const int E = f.E, ER = imax(f.RL.e, f.RR.e);
    const i64 DL = f.SL < 0 ? f.SL : 0, DR = f.SR > 0 ? f.SR : 0;
    int lz;
    const i64 iD = rcp(DR - DL, lz);
    const i64 one = 1LL << 60;
    i64 a = mulk<0, 2>(DR << (lz - 2), iD);  // units of 2^-60
    a = f.SL >= 0 ? one : (f.SR <= 0 ? 0 : a);
    const i64 b = one - a;
    const i64 gL = f.uL - DL, gR = f.uR - DR;
    // a rho_L (u_L - D_L) and b rho_R (u_R - D_R), units 2^(ER + E - 59)
    const i64 A = mulk<2, 2>(a, mulk<0, 0>(f.RL.m, gL) >> imin(ER - f.RL.e, 63));
    const i64 B = mulk<2, 2>(b, mulk<0, 0>(f.RR.m, gR) >> imin(ER - f.RR.e, 63));
    Fm = to_double(A + B, ER + E - 59);
    // a p_L and b p_R, units 2^(ER + 2E - 60); over gamma - 1 with G.room bits of room
    const int sp = ER + 2 * E;
    const i64 pL = mulk<2, 2>(a, f.PL.m >> imin(sp + 2 - f.PL.e, 63));
    const i64 pR = mulk<2, 2>(b, f.PR.m >> imin(sp + 2 - f.PR.e, 63));
    Fn = to_double(mulk<2, 2>(A, f.uL) + mulk<2, 2>(B, f.uR) + pL + pR, ER + 2 * E - 60);
    const i64 TL = mulk<2, 1>(A, s.vL), TR = mulk<2, 1>(B, s.vR);
    Ft = to_double(TL + TR, ER + E + X.t - 59, bad);
    // energy: p (u - D) / (gamma - 1) + p u + rho (u - D) (u^2 + v^2) / 2, units
    // 2^(ER + 3E - 62 + room)
    const i64 qL = mulk<2, 2>(a, sra(mulk<0, 0>(f.PL.m, G.gi), sp - f.PL.e - G.gie + G.room));
    const i64 qR = mulk<2, 2>(b, sra(mulk<0, 0>(f.PR.m, G.gi), sp - f.PR.e - G.gie + G.room));
    const int z = clz32((uint32_t)(hi32(qL) | hi32(qR))) - 1;
    const i64 h = mulk<0, 1>(qL << z, gL) + mulk<0, 1>(qR << z, gR);
    const i64 t = mulk<1, 1>(TL, s.vL) + mulk<1, 1>(TR, s.vR);
    // a faster flow along the face sets the unit, rr bits above
    const int st = 2 * (E - X.t) - 3, rr = imax(-st, 0);
    if (!fits(iabs(h), z - 4 + rr)) return false;
    const i64 k = mulk<2, 2>(A, mulk<2, 2>(f.uL, f.uL)) + mulk<2, 2>(B, mulk<2, 2>(f.uR, f.uR)) +
                  mulk<3, 2>(pL, f.uL) + mulk<3, 2>(pR, f.uR);
    Fe = to_double(shift(h, z - 4 + rr) + (sra(k, rr) + shift(t, st + rr) >> G.room),
                   ER + 3 * E - 62 + G.room + rr);
    return (int32_t)bad >= 0;
}

// The flux (HLL or HLLC) and the larger wave speed of one face given by its two states, {rho, p,
// normal, tangential velocity}; false where the integer solver does not take it.
template <bool HLL>
GD_HD bool euler_flux(const i64* a, const i64* b, const int* top, const Gas& G, double* F,
                      double& UU, bool& speed, bool speed_only) {
    const Tops X{top[0], top[1], top[2], top[3]};
    const States s{a[0], b[0], a[1], b[1], a[2], b[2], a[3], b[3]};
    const Fan f = fan_of<HLL>(s, X, G, UU);
    speed = f.ok;
    if (!f.ok) return false;
    if (speed_only) return true;
    return HLL ? hll(f, s, X, G, F[0], F[1], F[2], F[3]) : hllc(f, s, X, G, F[0], F[1], F[2], F[3]);
}
template <bool HLL>
GD_HD bool euler_face(const double* L, const double* R, const Gas& G, double* F, double& UU) {
    i64 q[8], a[4], b[4];
    Keys<4> k[2];
    int top[4];
    bool speed;
    cell_units<4>(L, q, 1, k[0]);
    cell_units<4>(R, q + 4, 1, k[1]);
    return G.room >= 0 && face_states<4, 1>(q + 4, 4, 1, k + 1, 1, true, a, b, top) &&
           euler_flux<HLL>(a, b, top, G, F, UU, speed, false);
}

}  // namespace fx
}  // namespace gd
