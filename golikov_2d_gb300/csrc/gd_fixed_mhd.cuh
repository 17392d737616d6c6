// gd_fixed_mhd.cuh -- the HLLD and HLLC-MHD face fluxes in scaled 64-bit integers (see
// gd_fixed.cuh).
//
// The states, speeds and guards of hlld_local (gd_mhd_flux.cuh; Gas_Dinamic.cu:964-1510), with
// the fluxes of the star states in the form the jump conditions across S_K give them.  K is the
// side the flux is taken from, m = rho (S - u), q = S_M / (S - S_M), b the HLL mean normal field:
//   mass F = rho q (S - u), normal momentum F S_M + p_T* - b_K^2, p_T* = p_T + m (S_M - u),
//   tangential F v* + m (v* - v) - b_K b_t, field S b* - (S - u) b_t - v b_K,
//   energy q (S - u) (p gamma / (gamma - 1) + rho (u^2 + v^2) / 2 + |b|^2 + rho S (S_M - u))
//          + b (q (v.b - v*.b*) - v*.b*) + (b - b_K) v.b,
// and S** (U** - U*) on top between the Alfven waves.  Only K's star state is formed unless the
// face lies between the Alfven waves.  HLLC-MHD (Gas_Dinamic.cu:1137-1302) is the same with v*, b*
// and v*.b* of the HLL state of the fan, which the two sides' m and iS = 1 / (S_R - S_L) give:
//   b_t* = [(S_R - u_R) b_t,R + v_R b_R - (L)] iS,  v* = [m_R v_R + b_R b_t,R - (L)] / (m_R - m_L).
//
// Units: velocities 2^(E - 61) as for HLLC; fields 2^(X.b - 61), below 2^60 (tangential ones in units
// of their own, see FanM); rho v^2 quantities
// 2^(ER + 2E - 59) and 2^(ER + 2E - 60), ER the larger density's exponent.  Squares of the field
// move to those by a shift: |b|^2 / 2 <= rho c_f^2 bounds them there.
#pragma once

#include "gd_fixed.cuh"

namespace gd {
namespace fx {

// Exponents of a face's units: densities, pressures, velocities and fields are in units of
// 2^(X - 61), below 2^62; b is the largest field's, and the normal field is below 2^60 in units of
// 2^(X.bn - 61).
struct TopsM {
    int r, p, n, t, b, bn, bt, bz;
};
struct StatesM {
    i64 r, p, un, ut, bn, bt, bz;
};
struct FluxI {
    double m, mn, mt, e, bn, bt, bz;
};

// |x| < 2^61 (and a little beyond on the negative side)
GD_HD bool below61(i64 x) { return (uint32_t)(hi32(x) + (1 << 29)) < (1u << 30); }

// sqrt(x) 2^(29 + h) of x 2^(2 h) in [2^61, 2^63): the root (w, in [2^59, 2^61)) and, where asked,
// the reciprocal root times 2^(91 - h).  As sqrt_over: e = 1 - x y^2 for the FP32 seed y.
template <bool RECIP>
GD_HD i64 sqrt_norm(i64 x, i64& rs) {
    const uint32_t y = (uint32_t)(rsqrt_seed((float)hi32(x)) * 35184363700224.0f);  // 2^45 - 2^23
    const i64 w = mul32(x, y);
    const i64 e = (1LL << 58) - mul32(w, y);
    const int32_t es = (int32_t)(e >> 15);
    const i64 g = (e << 3) + (wide(es, 3 * es) >> 27);
    if (RECIP) rs = ((i64)((u64)y << 30)) + mul32(g, y);
    return w + (mulk<0, 0, false>(w, g << 21) >> 19);
}
// sqrt(x) 2^31 for 0 <= x < 2^63
GD_HD i64 sqrt31(i64 x) {
    const int z = (clz64((u64)x) - 1) & ~1;
    i64 none;
    const i64 w = sqrt_norm<false>((i64)((u64)x << z), none);
    return (w << 2) >> (z >> 1);
}

// What a side gives: density, pressure, |b|^2 and b_n^2 in units of 2^(2 X.b - 58), and the fast
// speed w 2^(k - 60).
struct SideM {
    Pos R, P;
    i64 bb, n2, w;
    int k;
};
GD_HD SideM side_of(const StatesM& s, const TopsM& X, const Gas& G) {
    SideM S;
    S.R = pos_of(s.r, X.r);
    S.P = pos_of(s.p, X.p);
    S.n2 = mulk<0, 0>(s.bn, s.bn);
    const i64 t2 = mulk<0, 0>(s.bt, s.bt) + mulk<0, 0>(s.bz, s.bz);
    S.bb = S.n2 + t2;
    // gamma p, |b|^2 and the tangential part in one unit 2^U, below 2^61 and the larger above 2^59
    const i64 gp = mulk<0, 0>(S.P.m, G.g);
    const int ug = S.P.e + G.ge - 60;
    const int z = clz32((uint32_t)hi32(S.bb)) - 2;
    const int ub = 2 * X.b - 58 - z;
    const int U = imax(ug, ub) + 1;
    const i64 g1 = gp >> imin(U - ug, 63);
    const int sb = imin(U - ub, 63);
    const i64 b1 = (S.bb << z) >> sb, t1 = (t2 << z) >> sb;
    // a^2 - 4 gamma p b_n^2 with a = gamma p + |b|^2, as a sum: four times it
    const i64 d = g1 - b1;
    const i64 disc = mulk<1, 1>(d, d) + mulk<2, 2>(g1, t1);
    const i64 x = (g1 + b1 + sqrt31(disc)) >> 1;
    const int lz = clz32((uint32_t)hi32(x));
    S.w = sqrt_over(x << (lz - 2), U - lz + 62, S.R, S.k);
    return S;
}

// The star state of one side: v - v0, w, b_t, b_z behind the fast wave (Gas_Dinamic.cu:1306-1350).
// am = |rho (S - u)|, ad = |S - S_M|, as = |S - u|; bn2 the square of the mean normal field in
// units of 2^(ER + 2E - 59), st and sh the shifts that bring products of two fields to them (to the
// tangential velocity's where one is tangential), thr the guard's 1e-5 in them.  False where a ratio leaves its range.
struct StarM {
    i64 dv, dw, bt, bz;
};
GD_HD bool star_of(i64 am, i64 ad, i64 as, i64 SMu, i64 bn, i64 bn2, int st, int sh, i64 thr,
                   i64 bt, i64 bz, StarM& T) {
    const i64 tt = mulk<2, 1>(am, ad) - bn2;
    const i64 at = iabs(tt);
    if (at < thr) {
        T.dv = T.dw = T.bt = T.bz = 0;
        return true;
    }
    if (hi32(at) == 0) return false;
    int lz;
    const i64 it = rcp(at, lz);
    const i64 num = mulk<2, 1>(am, as) - bn2;
    const i64 x1 = shift(mulk<0, 0>(bn, bt), st), x2 = shift(mulk<0, 0>(bn, bz), sh);
    // The ratios to at, up to 2^r: r > 0 towards the speeds where the Alfven and the fast wave meet.
    // Beyond 4 the cancellation in at costs the ratios more digits than in binary64.
    const i64 top = iabs(num >> 1) | iabs(x1) | iabs(x2);
    const int r = imax(lz - clz32((uint32_t)hi32(top)) + 1, 0);
    const i64 k1 = mulk<0, 2>((x1 >> r) << (lz - 2), it), k2 = mulk<0, 2>((x2 >> r) << (lz - 2), it);
    const i64 d = mulk<0, 2>((num >> 1 >> r) << (lz - 2), it);
    const i64 dv = mulk<2, 1>(k1, SMu), dw = mulk<2, 1>(k2, SMu);
    const i64 ct = mulk<2, 1>(d, bt), cz = mulk<2, 1>(d, bz);
    if (r > 2 || (r > 0 && !(fits(iabs(dv) | iabs(dw), -r - 1) && fits(iabs(ct) | iabs(cz), -r - 2))))
        return false;
    const bool neg = tt < 0;
    T.dv = (neg ? dv : -dv) << (1 + r);
    T.dw = (neg ? dw : -dw) << (1 + r);
    T.bt = (neg ? -ct : ct) << (2 + r);
    T.bz = (neg ? -cz : cz) << (2 + r);
    return true;
}

// rho* = am / ad, and its root s 2^(k - 60) (and reciprocal root rs 2^(-60 - k))
GD_HD Pos star_density(i64 am, i64 iad, int lz, int ER) {
    const i64 t = mulk<2, 2>(am, iad);
    const int z = clz32((uint32_t)hi32(t));
    return Pos{t << (z - 1), ER + lz - z + 1};
}
template <bool RECIP>
GD_HD i64 root_of(Pos R, int& k, i64& rs) {
    const int odd = R.e & 1;
    k = (R.e + odd) >> 1;
    return sqrt_norm<RECIP>(R.m >> odd, rs);
}

// The larger wave speed of the face between A and B, and all speeds.
//
// Tangential components may be far below the normal ones and are carried by them, so they have
// units of their own: tangential velocities 2^(E - 61 - tv), tangential fields 2^(X.b - 61 - tb),
// and the z field and velocity 2^(X.b - 61 - z) and 2^(E - 61 - z).  Every flux is linear in each
// pair, or has products of two of it, which shift back.  A normal field couples velocity and field:
// both units then follow the larger of v and b / sqrt(rho), 2^(-sh/2) of the speed per unit of the
// field, up to the bits by which the normal field's own speed is below the fan's (what v adds to the
// field's flux, and b to the momentum's, is that much less).  kRoom bits are left above the
// components, for star states above them.
//
// A flow along the face far faster than its waves would set the unit of all speeds and cost the fan
// its digits.  The fluxes follow a change of frame exactly, so the face is solved in a frame that
// moves along it with w, one side's tangential velocity to 52 bits (units 2^(X.t - 61); 0 in all
// other faces), and mhd_flux adds w's momentum, energy and induction.
constexpr int kRoom = 3;
struct FanM {
    SideM A, B;
    i64 uA, uB, vA, vB, SL, SR, w;
    int E, ER, kmin, tv, tb, z, nb;
    int sh;  // what brings products of two fields to units of 2^(ER + 2E - 59)
    bool ok;
};
GD_HD FanM fan_of(StatesM& a, StatesM& b, const TopsM& X, const Gas& G, double& UU) {
    FanM f;
    const int bt = X.b - X.bt, bz = X.b - X.bz;
    f.nb = X.b - X.bn;
    f.A = side_of(StatesM{a.r, a.p, a.un, a.ut, asr(a.bn, f.nb), asr(a.bt, bt), asr(a.bz, bz)}, X, G);
    f.B = side_of(StatesM{b.r, b.p, b.un, b.ut, asr(b.bn, f.nb), asr(b.bt, bt), asr(b.bz, bz)}, X, G);
    const int kmax = imax(f.A.k, f.B.k);
    f.kmin = imin(f.A.k, f.B.k);
    f.ER = imax(f.A.R.e, f.B.R.e);
    f.E = imax(kmax + 2, scale_of(a.un, b.un, X.n));
    int xv = scale_of(a.ut, b.ut, X.t);
    f.w = 0;
    if (xv > f.E + 1) {
        f.w = a.ut & ~1023LL;
        a.ut -= f.w;
        b.ut -= f.w;
        xv = top_of(a.ut, b.ut, X.t);
    }
    f.E = imax(f.E, xv);
    const int dr = f.A.R.e - f.B.R.e;
    f.ok = kmax - f.kmin <= 2 && f.E - kmax <= 24 && (uint32_t)(dr + 3) <= 6u;
    if (!f.ok) return f;
    const i64 cA = f.A.w >> (f.E - 1 - f.A.k), cB = f.B.w >> (f.E - 1 - f.B.k);
    const i64 c = cA > cB ? cA : cB;
    f.uA = asr(a.un, f.E - X.n);
    f.uB = asr(b.un, f.E - X.n);
    f.tv = imax(f.E - xv - kRoom, 0);
    f.tb = imax(X.b - scale_of(a.bt, b.bt, X.bt) - kRoom, 0);
    f.z = imax(X.b - scale_of(a.bz, b.bz, X.bz) - kRoom, 0);
    f.sh = f.ER + 2 * f.E - 1 - 2 * X.b;
    if ((a.bn | b.bn) != 0) {
        const int h = imax(f.sh, 0) >> 1, tv = f.tv;
        const int k = imax(h + f.nb - 2, 0);
        f.tv = imin(tv, f.tb + h + k);
        f.tb = imin(imin(f.tb, imax(tv - h, 0) + k), f.tv + f.nb);
    }
    f.vA = shift(a.ut, f.E - X.t - f.tv);
    f.vB = shift(b.ut, f.E - X.t - f.tv);
    a.bt = asr(a.bt, bt - f.tb);
    b.bt = asr(b.bt, bt - f.tb);
    a.bz = asr(a.bz, bz - f.z);
    b.bz = asr(b.bz, bz - f.z);
    f.SL = (f.uA < f.uB ? f.uA : f.uB) - c;
    f.SR = (f.uA > f.uB ? f.uA : f.uB) + c;
    UU = to_double(-f.SL > f.SR ? -f.SL : f.SR, f.E - 61);
    return f;
}

// m 2^(e - 62) in units of 2^u, at least 1, or the largest integer where it does not fit
GD_HD i64 threshold(i64 m, int e, int u) {
    const int s = u - e + 62;
    return s < 0 ? 0x7fffffffffffffffLL : (m >> imin(s, 62)) | 1;
}

// x << (lz - 2) fits, x >= 0
GD_HD bool scales(i64 x, int lz) { return x >> imin(65 - lz, 63) == 0; }

// At a mirror the contact stands on the face, and the flux may jump from one side's to the other's;
// binary64 finds S_M = 0 there exactly and takes the side below.  Products here round down, so that
// S_M's numerator comes out as 0 to some units (2^(ER + 2E - 60)): the side below is taken down to
// -kTie, 2^-54 of rho c^2 and the size of binary64's own roundings.  (Setting such a numerator to 0
// says the same and took 1.95 ms for four steps of 1024^2 where this takes 1.89.)
constexpr i64 kTie = 32;

template <bool HLLD>
GD_HD bool mhd_flux(const FanM& f, const StatesM& a, const StatesM& b, const TopsM& X, const Gas& G,
                    FluxI& F) {
    const int E = f.E, ER = f.ER, XB = 2 * X.b;
    const i64 suA = f.SL - f.uA, suB = f.SR - f.uB;
    const i64 mA = mulk<0, 0>(f.A.R.m, suA) >> (ER - f.A.R.e);
    const i64 mB = mulk<0, 0>(f.B.R.m, suB) >> (ER - f.B.R.e);
    // total pressures in units of 2^(ER + 2E - 60)
    const int sp = ER + 2 * E + 2, sq = f.sh;
    const i64 ptA = (f.A.P.m >> imin(sp - f.A.P.e, 63)) + shift(f.A.bb, sq);
    const i64 ptB = (f.B.P.m >> imin(sp - f.B.P.e, 63)) + shift(f.B.bb, sq);
    const i64 N = mulk<1, 3>(mB, f.uB) - mulk<1, 3>(mA, f.uA) + (ptA - ptB);
    int lz;
    const i64 iD = rcp(mB - mA, lz);
    i64 SM = mulk<0, 2>(N << (lz - 2), iD);
    // the mean normal field
    int lzs;
    const i64 iS = rcp(f.SR - f.SL, lzs);
    const i64 bs = mulk<2, 1>(f.SR, b.bn) - mulk<2, 1>(f.SL, a.bn);
    i64 bn = mulk<0, 2>(bs << (lzs - 2), iS) << 1;

    const bool takeL = f.SL >= 0 || N >= -kTie;
    const bool star = takeL ? f.SL < 0 : f.SR > 0;
    const Pos R{takeL ? f.A.R.m : f.B.R.m, takeL ? f.A.R.e : f.B.R.e};
    const Pos Pk{takeL ? f.A.P.m : f.B.P.m, takeL ? f.A.P.e : f.B.P.e};
    const i64 bbK = takeL ? f.A.bb : f.B.bb, n2K = takeL ? f.A.n2 : f.B.n2;
    const i64 un = takeL ? f.uA : f.uB, ut = takeL ? f.vA : f.vB;
    const i64 bnK = takeL ? a.bn : b.bn, btK = takeL ? a.bt : b.bt, bzK = takeL ? a.bz : b.bz;
    const i64 m = takeL ? mA : mB, ptK = (takeL ? ptA : ptB) >> 1;
    const i64 S = takeL ? f.SL : f.SR, su = takeL ? suA : suB;

    // of products of the normal field with itself, the z field and a tangential one, to momenta; and
    // with a tangential velocity, to the tangential field's flux
    const int nb = f.nb, sn = f.sh + nb, st = sn - (f.tv - f.tb), dn = f.tv - f.tb + nb;
    const int vb = f.tv + f.tb;
    // units 2^(E + X.b - 61)
    const i64 ub = asr(mulk<2, 1>(un, bnK), nb) + asr(mulk<2, 1>(ut, btK), vb);
    i64 qs = un, qsg = 0, sb = ub, S2 = 0;
    StarM K{0, 0, btK, bzK};
    Pos RK = R;
    i64 sK = 0, am = 0, bn2 = 0, thr = 0;
    int kK = 0;
    bool alfven = false;
    if (star) {
        if (E - f.kmin > 4) return false;
        const i64 ad = takeL ? SM - S : S - SM;
        if (hi32(ad) <= 0) return false;
        int lza;
        const i64 iA = rcp(ad, lza);
        const i64 q = mulk<0, 2>(SM << (lza - 2), iA);
        qsg = takeL ? -q : q;  // S_M / (S - S_M), at most 1 in size, in units of 2^-60
        qs = mulk<2, 1>(qsg, su) << 1;
        if constexpr (HLLD) {
            am = iabs(m);
            bn2 = shift(mulk<0, 0>(bn, bn), sn + nb);
            thr = threshold(0x53e2d6238da3c211LL, -17, ER + 2 * E - 59);  // 1e-5
            if (!star_of(am, ad, iabs(su), SM - un, bn, bn2, st, sn, thr, btK, bzK, K)) return false;
            RK = star_density(am, iA, lza, ER);
            i64 rs;
            sK = root_of<true>(RK, kK, rs);
            const i64 abn = iabs(bn);
            // |b| / sqrt(rho*), where |b| > 1e-6 (Gas_Dinamic.cu:1352-1369)
            const bool va0 = abn <= threshold(0x431bde82d7b634daLL, -20, X.bn - 61);
            const i64 va = va0 ? 0 : shift(mulk<1, 2>(abn, rs), kK + E - 1 - X.bn);
            S2 = takeL ? SM - va : SM + va;
            alfven = !va0 && (takeL ? S2 < 0 : S2 > 0);
        } else {
            // the fan's HLL state: v*, b*, and v*.b* with its own u and w
            const i64 nA = f.A.n2, nB = f.B.n2;  // b_n^2
            const i64 tA = mulk<0, 0>(a.bn, a.bt), tB = mulk<0, 0>(b.bn, b.bt);
            const i64 zA = mulk<0, 0>(a.bn, a.bz), zB = mulk<0, 0>(b.bn, b.bz);
            const i64 N1 = N + (shift(nB - nA, sq) << 1);
            const i64 N2 = mulk<1, 3>(mB, f.vB) - mulk<1, 3>(mA, f.vA) + (shift(tB - tA, st) << 1);
            const i64 N3 = shift(zB - zA, sn) << 1;
            i64 Tt = mulk<1, 2>(suB, b.bt) - mulk<1, 2>(suA, a.bt) +
                     asr(mulk<2, 1>(f.vB, b.bn) - mulk<2, 1>(f.vA, a.bn), dn);
            const i64 Tz = mulk<1, 2>(suB, b.bz) - mulk<1, 2>(suA, a.bz);
            if (f.w != 0) {  // the one term that a jump of the normal field keeps out of the frame
                const i64 wb = mulk<1, 1>(f.w, b.bn - a.bn);
                const int sw = E - f.tb - X.t - 1 + nb;
                if (!fits(iabs(wb), sw)) return false;
                Tt += shift(wb, sw);
            }
            if (!(scales(iabs(N1) | iabs(N2) | iabs(N3), lz) &&
                  scales(iabs(Tt) | iabs(Tz), lzs)))
                return false;
            const i64 u1 = mulk<0, 2>(N1 << (lz - 2), iD), vs = mulk<0, 2>(N2 << (lz - 2), iD);
            const i64 ws = mulk<0, 2>(N3 << (lz - 2), iD);
            K.bt = mulk<0, 2>(Tt << (lzs - 2), iS) << 1;
            K.bz = mulk<0, 2>(Tz << (lzs - 2), iS) << 1;
            K.dv = vs - ut;
            if (!(below61(u1) && below61(ws) && below61(vs) && below61(K.bt) && below61(K.bz)))
                return false;
            sb = asr(mulk<2, 1>(u1, bn), nb) + asr(mulk<2, 1>(vs, K.bt), vb) +
                 asr(mulk<2, 1>(ws, K.bz), 2 * f.z);
        }
    } else {  // the physical flux of K: no mean of both sides in it
        SM = un;
        bn = bnK;
    }
    const i64 SMu = SM - un, vK = ut + K.dv;
    if (!(below61(vK) && below61(K.dw) && below61(K.bt) && below61(K.bz))) return false;
    if (HLLD && star)
        sb = asr(mulk<2, 1>(SM, bn), nb) + asr(mulk<2, 1>(vK, K.bt), vb) +
             asr(mulk<2, 1>(K.dw, K.bz), 2 * f.z);

    const int32_t qh = hi32(qs);
    const int z = clz32((uint32_t)(qh ^ (qh >> 31))) - 1;
    const i64 qn = qs << z;
    const i64 M = mulk<0, 0>(R.m, qn);
    const int em = R.e + E - 59 - z;
    F.m = to_double(M, em);
    const int dR = ER - R.e;
    const i64 n2s = shift(n2K, sq), bnt = shift(mulk<0, 0>(bnK, btK), st);
    const i64 mn = ptK + (mulk<1, 2>(M, SM) >> imin(z + dR, 63)) + mulk<2, 1>(m, SMu) - n2s;
    i64 mt = (mulk<1, 2>(M, vK) >> imin(z + dR, 63)) + mulk<2, 1>(m, K.dv) - bnt;
    i64 ft = mulk<2, 1>(S, K.bt) - mulk<1, 2>(su, btK) - asr(mulk<2, 1>(ut, bnK), dn);
    i64 fz = mulk<2, 1>(S, K.bz) - mulk<1, 2>(su, bzK);
    const i64 H = mulk<1, 1>(un, un) + asr(mulk<1, 1>(ut, ut), 2 * f.tv) + mulk<2, 1>(S, SMu);
    const i64 B = sra(mulk<0, 0>(Pk.m, G.gg), ER + 2 * E - Pk.e - G.gge + G.room) +
                  ((mulk<0, 1>(R.m, H) >> dR) + shift(bbK, ER + 2 * E - 2 - XB) >> G.room);
    const i64 y = (mulk<2, 1>(qsg, ub - sb) << 1) - sb;
    // units 2^(ER + 3E - 61)
    const i64 e0 = mulk<0, 2>(qn, B);
    if (!(below61(B) && fits(iabs(e0), z - 2 - G.room))) return false;
    i64 e = shift(e0, z - 2 - G.room) +
            shift(mulk<2, 0>(bn, y) + mulk<2, 0>(bn - bnK, ub), sn);

    i64 dm = 0;
    if (HLLD && alfven) {
        // the other side's star state and the states between the Alfven waves
        // (Gas_Dinamic.cu:1371-1430); v3 = vO + w (vK - vO) + ..., w = sK / (sK + sO)
        const i64 unO = takeL ? f.uB : f.uA, utO = takeL ? f.vB : f.vA;
        const i64 btO = takeL ? b.bt : a.bt, bzO = takeL ? b.bz : a.bz;
        const i64 amO = iabs(takeL ? mB : mA), asO = iabs(takeL ? suB : suA);
        const i64 adO = takeL ? f.SR - SM : SM - f.SL;
        if (hi32(adO) <= 0) return false;
        StarM O;
        if (!star_of(amO, adO, asO, SM - unO, bn, bn2, st, sn, thr, btO, bzO, O)) return false;
        const i64 vO = utO + O.dv;
        if (!(below61(vO) && below61(O.dw) && below61(O.bt) && below61(O.bz))) return false;
        int lzO, kO, lzt;
        const i64 iO = rcp(adO, lzO);
        i64 none;
        const i64 sO = root_of<false>(star_density(amO, iO, lzO, ER), kO, none);
        const int kk = imax(kK, kO) + 1;
        const i64 aK = sK >> imin(kk - kK, 63), aO = sO >> imin(kk - kO, 63);
        const i64 iT = rcp(aK + aO, lzt);
        const i64 w = mulk<0, 2>(aK << (lzt - 2), iT);
        const bool flip = takeL != (bn > 0);  // sign of b times that of O - K in R - L
        const int sv = E + kk + 3 - lzt - X.b;
        const i64 xt0 = mulk<1, 2>(O.bt - K.bt, iT);
        const int dt = f.tv - f.tb;
        const i64 xz = shift(mulk<1, 2>(O.bz - K.bz, iT), sv);
        // root(rho) times the jump of v may be far above a weak field, and the other way round
        if (!fits(iabs(xt0), sv - dt)) return false;
        const i64 xt = shift(xt0, sv - dt);
        const i64 v3 = vO + (mulk<2, 1>(w, vK - vO) << 1) + (flip ? -xt : xt);
        const i64 w3 = O.dw + (mulk<2, 1>(w, K.dw - O.dw) << 1) + (flip ? -xz : xz);
        const i64 wo = mulk<2, 2>(w, aO);
        const int sc = X.b - kk - E - 1;
        const i64 ct = mulk<2, 1>(wo, vO - vK), cz = mulk<2, 1>(wo, O.dw - K.dw);
        if (!(fits(iabs(ct), sc + dt) && fits(iabs(cz), sc))) return false;
        const i64 yt = shift(ct, sc + dt), yz = shift(cz, sc);
        const i64 bt3 = K.bt + (mulk<2, 1>(w, O.bt - K.bt) << 1) + (flip ? -yt : yt);
        const i64 bz3 = K.bz + (mulk<2, 1>(w, O.bz - K.bz) << 1) + (flip ? -yz : yz);
        if (!(below61(v3) && below61(w3) && below61(bt3) && below61(bz3) && below61(S2)))
            return false;
        const i64 sb3 = asr(mulk<2, 1>(SM, bn), nb) + asr(mulk<2, 1>(v3, bt3), vb) +
                        asr(mulk<2, 1>(w3, bz3), 2 * f.z);
        dm = shift(mulk<2, 1>(mulk<0, 0>(RK.m, S2), v3 - vK), ER - RK.e);
        mt += dm;
        ft += mulk<2, 1>(S2, bt3 - K.bt);
        fz += mulk<2, 1>(S2, bz3 - K.bz);
        const i64 de = shift(mulk<1, 2>(mulk<2, 0>(sK, sb - sb3), S2), ER + E - kK - X.b - 2);
        e += flip ? de : -de;
    }
    uint32_t bad = 0;
    F.mn = to_double(mn, ER + 2 * E - 59);
    F.mt = to_double(mt, ER + 2 * E - 59 - f.tv, bad);
    F.e = to_double(e, ER + 3 * E - 61);
    F.bt = to_double(ft, E + X.b - 61 - f.tb, bad);
    F.bz = to_double(fz, E + X.b - 61 - f.z, bad);
    if (f.w != 0) {
        // what w multiplies in the energy flux: the momentum flux, but for guarded star states
        const i64 yt = (mulk<2, 1>(qsg, btK - K.bt) << 1) - K.bt;
        const i64 et = (mulk<1, 2>(M, ut) >> imin(z + dR, 63)) + dm +
                       shift(mulk<0, 0>(bn, yt) + mulk<0, 0>(bn - bnK, btK), st);
        const double w = to_double(f.w, X.t - 61), et_d = to_double(et, ER + 2 * E - 59 - f.tv, bad);
        F.e = std::fma(w, std::fma(0.5 * w, F.m, et_d), F.e);
        F.mt = std::fma(w, F.m, F.mt);
        F.bt = std::fma(-w, to_double(bnK, X.bn - 61, bad), F.bt);
    }
    return (int32_t)bad >= 0;
}

// The flux and the larger wave speed of a face from its states and their exponents (face_states);
// speed: whether the latter is valid.
template <bool HLLD>
GD_HD bool mhd_face_flux(const i64* p, const i64* q, const int* top, const Gas& G, FluxI& F,
                         double& UU, bool& speed, bool speed_only) {
    const int e4 = scale_of(p[4], q[4], top[4]), e5 = scale_of(p[5], q[5], top[5]);
    const int e6 = scale_of(p[6], q[6], top[6]);
    const TopsM X{top[0], top[1], top[2], top[3], imax(imax(e4, e5), e6), e4, top[5], top[6]};
    StatesM a{p[0], p[1], p[2], p[3], asr(p[4], e4 - top[4]), p[5], p[6]};
    StatesM b{q[0], q[1], q[2], q[3], asr(q[4], e4 - top[4]), q[5], q[6]};
    const FanM f = fan_of(a, b, X, G, UU);
    speed = f.ok;
    if (!f.ok) return false;
    if (speed_only) return true;
    // the normal field's flux in its own unit, cut at 2^-1020
    const int un = f.E + top[4] - 60, low = imax(-1020 - un, 0);
    const i64 S = -f.SL > f.SR ? -f.SL : f.SR;
    F.bn = to_double(asr(mulk<2, 0>(S, p[4] - q[4]), low), un + low);
    return mhd_flux<HLLD>(f, a, b, X, G, F);
}
// The two states {rho, p, un, ut, bn, bt, bz} of a face in units of their own; false where the
// integer solver does not take them.
GD_HD bool face_units(const double* L, const double* R, const Gas& G, i64* a, i64* b, int* top) {
    i64 q[14];
    Keys<7> k[2];
    cell_units<7>(L, q, 1, k[0]);
    cell_units<7>(R, q + 7, 1, k[1]);
    return G.room >= 0 && face_states<7, 1>(q + 7, 7, 1, k + 1, 1, true, a, b, top);
}
// Flux and larger wave speed of that face.
template <bool HLLD>
GD_HD bool mhd_face(const double* L, const double* R, const Gas& G, FluxI& F, double& UU) {
    i64 a[7], b[7];
    int top[7];
    bool speed;
    return face_units(L, R, G, a, b, top) &&
           mhd_face_flux<HLLD>(a, b, top, G, F, UU, speed, false);
}

}  // namespace fx
}  // namespace gd
