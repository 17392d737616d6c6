// gd_adjoint.cu -- hand-written discrete adjoint (reverse mode, VJP) of the fast MHD step.
//
// The step U' = S(U; dt) of gd_fast_mhd.cu (HLLD, minmod TVD, Powell source, Cartesian,
// periodic) is differentiated with dt held fixed and every non-smooth choice (minmod
// selection, wave-speed min/max, region selection, guards, floors) frozen at the branch
// the forward values take.  Given lambda' = dL/dU', one reverse step returns
// lambda = dL/dU = S'(U)^T lambda' in two passes:
//
//   A  per cell (adj_update_kernel): the transpose of the cell update.  Inputs: U, the
//      forward flux differences d[7] and the Powell term divb of that cell (stored by the
//      recompute pass), lambda'.  Outputs: the direct adjoint of the cell state, the adjoint
//      of d[7] and of divb.
//   B  per face, then per cell (adj_face_kernel, adj_gather_kernel): every face recomputes
//      its forward states and the flux's star states and runs the flux's reverse sweep on
//      Fbar = k (dbar_low - dbar_high); the adjoints of the two face states are gathered
//      into the cells through the reconstruction (c +- slope/2, minmod choice, rho/p
//      fallback) and the Powell central difference, in a fixed order (deterministic).
//
// All internal arithmetic is in Heaviside-Lorentz field units (b = B / sqrt(4 pi)), as in
// the forward kernel; adjoints w.r.t. the stored Gaussian field are converted at the ends.
#include "gd_internal.cuh"
#include "gd_kernels.h"
#include "gd_mhd_flux.cuh"

namespace gd {
namespace {

constexpr int NF = 7;
constexpr int NT = 256;

// ---------------------------------------------------------------------------------------
// Pass A: transpose of the cell update (Cartesian).
// aux layout per cell: d[0..6] (slot order m, e, mx, my, bx, by, bz), divb.  Adjoint
// scratch per cell: qbar[0..6] (field order rho, p, vx, vy, bx, by, bz, field in b units),
// dbar[0..6] (slot order), divbbar.  Bound by the FP64 pipe: 40 us at 512^2, 49 us before the
// squares of both kinetic energies shared one factor (62 FP64 operations per cell, 100 before).
// ---------------------------------------------------------------------------------------
__global__ void __launch_bounds__(NT) adj_update_kernel(Params P, CPlanes U, const double* aux,
                                                        CPlanes lam_out, double* scratch) {
    const long long K = (long long)P.N * P.M;
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < K;
         k += (long long)gridDim.x * blockDim.x) {
        const double r = U.f[0][k], p = U.f[1][k], u = U.f[2][k], v = U.f[3][k];
        // rounded products, as the forward update has them (see ld_b)
        const double bx = imul(U.f[4][k], kInvSpi4), by = imul(U.f[5][k], kInvSpi4);
        const double bz = imul(U.f[6][k], kInvSpi4);
        double d[NF];
#pragma unroll
        for (int f = 0; f < NF; ++f) d[f] = aux[(size_t)f * K + k];
        const double divb = aux[(size_t)7 * K + k];
        // forward (same operations as the tile update)
        const double ub = fma(u, bx, imul(v, by));
        const double bb = fma(bz, bz, fma(by, by, imul(bx, bx)));
        const double V1 = fma(u, u, imul(v, v));
        const double K1 = fma(r, V1, bb);
        double r2 = r - d[0];
        const bool rfl = le_zero(r2);
        if (rfl) r2 = r;
        const double mx2 = fma(r, u, -fma(bx, divb, d[2]));
        const double my2 = fma(r, v, -fma(by, divb, d[3]));
        const double bx2 = bx - fma(u, divb, d[4]);
        const double by2 = by - fma(v, divb, d[5]);
        const double bz2 = bz - d[6];
        const double dE = fma(ub, divb, d[1]);
        const double inv = rcp_fast(r2);
        const double u2 = imul(mx2, inv), v2 = imul(my2, inv);
        const double V2 = fma(u2, u2, imul(v2, v2));
        const double K2 = fma(r2, V2, fma(bz2, bz2, fma(by2, by2, imul(bx2, bx2))));
        const double p2 = fma(P.hgm1, K1 - K2, fma(-P.gm1, dE, p));
        const bool pfl = le_zero(p2);
        // reverse.  p2 = p - gm1 dE + hgm1 (K1 - K2); gm1 = 2 hgm1 and r2 u2 = mx2 make one
        // factor w = gm1 p2b serve dE and every square of K1 and K2
        const double p2b = pfl ? 0.0 : lam_out.f[1][k];
        const double w = p2b * P.gm1, h = p2b * P.hgm1;
        const double u2b = fma(-w, mx2, lam_out.f[2][k]), v2b = fma(-w, my2, lam_out.f[3][k]);
        const double bx2b = fma(-w, bx2, imul(lam_out.f[4][k], kSpi4));
        const double by2b = fma(-w, by2, imul(lam_out.f[5][k], kSpi4));
        const double bz2b = fma(-w, bz2, imul(lam_out.f[6][k], kSpi4));
        // u2 = mx2 / r2, v2 = my2 / r2
        const double mx2b = imul(u2b, inv), my2b = imul(v2b, inv);
        const double r2b = fma(-mx2b, u2, fma(-my2b, v2, fma(-h, V2, lam_out.f[0][k])));
        const double db[NF] = {rfl ? 0.0 : -r2b, -w, -mx2b, -my2b, -bx2b, -by2b, -bz2b};
        const double pb = p2b;
        const double wr = w * r, wd = -w * divb;  // wd: adjoint of u . b
        const double rb = fma(mx2b, u, fma(my2b, v, fma(h, V1, r2b)));
        const double ub_ = fma(wr, u, fma(mx2b, r, fma(-bx2b, divb, wd * bx)));
        const double vb = fma(wr, v, fma(my2b, r, fma(-by2b, divb, wd * by)));
        const double bxb = fma(w, bx, fma(wd, u, fma(-mx2b, divb, bx2b)));
        const double byb = fma(w, by, fma(wd, v, fma(-my2b, divb, by2b)));
        const double bzb = fma(w, bz, bz2b);
        const double divbb =
            -fma(w, ub, fma(bx2b, u, fma(by2b, v, fma(mx2b, bx, my2b * by))));
        double* s = scratch;
        s[0 * K + k] = rb;
        s[1 * K + k] = pb;
        s[2 * K + k] = ub_;
        s[3 * K + k] = vb;
        s[4 * K + k] = bxb;
        s[5 * K + k] = byb;
        s[6 * K + k] = bzb;
#pragma unroll
        for (int f = 0; f < NF; ++f) s[(size_t)(7 + f) * K + k] = db[f];
        s[(size_t)14 * K + k] = divbb;
    }
}

// ---------------------------------------------------------------------------------------
// Reverse sweep of one HLLD face flux (method 3) in the local frame.
// Inputs: the two face states A (low) and B (high) as (r, p, un, ut, bn, bt, bz) and the
// adjoint of the flux (m, mn, mt, e, bn, bt, bz).  Writes the adjoints of A and B to Ab, Bb.
//
// The derivative is that of the forward's flux on the branch it takes; what is differentiated
// is the shortest form of that flux, not the forward's chain of operations.  K is the upwind
// side, O the other one, m = r (S - un), d = SM - un, D = S - SM, and X the state the flux
// belongs to (K's star state, or the double star).  The jump relations across S and across
// the Alfven wave hold identically for the solver's star formulas, so that with
// phi = rK SM and P* = pT + m d the flux is
//   m = phi,  mn = phi SM + P* - bnK^2,  mt = phi v - bn b + (bn - bnK) bt,
//   bt: SM b - bn v + (bn - bnK) ut,  bz: SM z - bn w,  e = SM (e + P*) - bn sb + (bn - bnK) wK
// with v, w, b, z, sb, e those of X.  Neither S nor the Alfven speeds appear any more; the
// other side's star state is needed for the double star alone; v* and b* of one wave share
// their reverse products; the reverse of a quotient n / q is that of n - q x = 0 (no chain
// through the reciprocal).  A side whose star guard fails (|tt| < 1e-5) has v* = ut and
// w* = b* = z* = 0; the three terms by which its flux then differs are added apart.
// ---------------------------------------------------------------------------------------
struct SideV {
    double r, p, un, ut, bn, bt, bz;
    double bn2, bb, pT, gp, a, disc, rq, rs, cf;  // rq = 1 / sqrt(disc), rs = 1 / sqrt(X r)
    bool disc0;
};

__device__ __forceinline__ void side_fwd(SideV& S, const double* q, const Params& P) {
    S.r = q[0]; S.p = q[1]; S.un = q[2]; S.ut = q[3]; S.bn = q[4]; S.bt = q[5]; S.bz = q[6];
    S.bn2 = imul<true>(S.bn, S.bn);
    S.bb = fma(S.bz, S.bz, fma(S.bt, S.bt, S.bn2));
    S.pT = fma(0.5, S.bb, S.p);
    S.gp = imul<true>(P.gamma, S.p);
    S.a = S.gp + S.bb;
    double disc = fma(S.a, S.a, imul<true>(imul<true>(-4.0, S.gp), S.bn2));
    S.disc0 = le_zero(disc);
    S.disc = S.disc0 ? 0.0 : disc;
    // sqrt_fast(disc) of the forward, keeping 1/sqrt(disc) for the reverse
    double sq;
    sqrt_and_rs_im<true>(S.disc, sq, S.rq);
    const double X = imul<true>(0.5, S.a + sq);
    // cf = sqrt_over(X, r) of the forward, keeping its 1/sqrt(X r) for the reverse
    sqrt_over_rs_im<true>(X, S.r, S.cf, S.rs);
}

// per-side adjoint accumulators of the face state and of two derived quantities
struct SideB {
    double r, p, un, ut, bn, bt, bz, pT, bb, bn2;
};

// adds k to the side the select names with one FP64 add (the other side is untouched)
__device__ __forceinline__ void add_to(bool first, double& a, double& b, double k) {
    const double s = (first ? a : b) + k;
    a = first ? s : a;
    b = first ? b : s;
}

// the side-generic tail: pT = 0.5 bb + p, bb = bz^2 + bt^2 + bn2, bn2 = bn^2
__device__ __forceinline__ void side_tail(const SideV& S, SideB& b, double* qb) {
    const double bbb = fma(0.5, b.pT, b.bb);
    const double bn2b = b.bn2 + bbb;
    qb[0] = b.r;
    qb[1] = b.p + b.pT;
    qb[2] = b.un;
    qb[3] = b.ut;
    qb[4] = fma(2.0 * bn2b, S.bn, b.bn);
    qb[5] = fma(2.0 * bbb, S.bt, b.bt);
    qb[6] = fma(2.0 * bbb, S.bz, b.bz);
}

// star state of one side: m, D = S - SM, d = SM - un as above, bbn = bn^2
struct StarV {
    double it, h, c, q;  // 1 / tt, d / tt, bn d / tt, 1 + m d / tt (all 0 where the guard fails)
    double v, w, b, z;
    bool g;
};

__device__ __forceinline__ StarV star_fwd(double m, double D, double d, double bn, double bbn,
                                          double ut, double bt, double bz) {
    StarV s;
    const double tt = fma(m, D, -bbn);
    s.g = mag_ge(tt, kMag1em5);
    s.it = s.g ? rcp_fast(tt) : 0.0;
    s.h = d * s.it;
    s.c = bn * s.h;
    s.q = s.g ? fma(m, s.h, 1.0) : 0.0;
    s.v = fma(-s.c, bt, ut);
    s.w = -s.c * bz;
    s.b = bt * s.q;
    s.z = bz * s.q;
    return s;
}

// its reverse: (vb, wb, bb, zb) onto the side's ut, bt, bz and onto m, D, d, bn
__device__ __forceinline__ void star_rev(const StarV& s, double m, double D, double bn, double bt,
                                         double bz, double vb, double wb, double bb, double zb,
                                         SideB& Q, double& mb, double& Db, double& db,
                                         double& bnb) {
    const double cb = fma(vb, bt, wb * bz);  // minus the adjoint of c
    const double qb = fma(bb, bt, zb * bz);
    Q.ut += vb;
    Q.bt = fma(bb, s.q, fma(-vb, s.c, Q.bt));
    Q.bz = fma(zb, s.q, fma(-wb, s.c, Q.bz));
    const double n = fma(qb, m, -cb * bn) * s.it;
    db += n;
    const double ttb = -n * s.h;
    mb = fma(ttb, D, fma(qb, s.h, mb));
    Db = fma(ttb, m, Db);
    bnb = fma(-2.0 * ttb, bn, fma(-cb, s.h, bnb));
}

// Fb = (m, mn, mt, e, bn, bt, bz); qa_b, qb_b receive (r, p, un, ut, bn, bt, bz).
__device__ __forceinline__ void hlld_vjp(const double* qa, const double* qb, const double* Fb,
                                         const Params& P, double* qa_b, double* qb_b) {
    SideV A, B;
    side_fwd(A, qa, P);
    side_fwd(B, qb, P);
    // ---- forward, shared part
    const bool minA = !dlt(B.un, A.un);              // uminN = A.un (else B.un)
    const bool maxB = dlt(A.un, B.un);               // umaxN = B.un (else A.un)
    const bool cfB = mag_lt(A.cf, B.cf);
    const double cmax = cfB ? B.cf : A.cf;
    const double SL = (minA ? A.un : B.un) - cmax, SR = (maxB ? B.un : A.un) + cmax;
    const double suL = SL - A.un, suR = SR - B.un;
    const double mL = A.r * suL, mR = B.r * suR;
    const double iden = rcp_fast(mR - mL);
    const double du = B.un - A.un;
    const double dA = fma(mR, du, A.pT - B.pT) * iden;  // SM - A.un
    const double SM = A.un + dA;
    const bool UUR = mag_lt(SL, SR);
    const bool takeL = ge_zero(SL) || ge_zero(SM);
    // the upwind side K and the other side O
    const double Kr = takeL ? A.r : B.r, Kp = takeL ? A.p : B.p;
    const double Kun = takeL ? A.un : B.un, Kut = takeL ? A.ut : B.ut;
    const double Kbn = takeL ? A.bn : B.bn, Kbt = takeL ? A.bt : B.bt;
    const double Kbz = takeL ? A.bz : B.bz, KpT = takeL ? A.pT : B.pT;
    const double Kbb = takeL ? A.bb : B.bb;
    const double Or = takeL ? B.r : A.r, Out = takeL ? B.ut : A.ut;
    const double Obn = takeL ? B.bn : A.bn, Obt = takeL ? B.bt : A.bt;
    const double Obz = takeL ? B.bz : A.bz;
    const double SK = takeL ? SL : SR, SO = takeL ? SR : SL;
    const double suK = takeL ? suL : suR, suO = takeL ? suR : suL;
    const double mK = takeL ? mL : mR, mO = takeL ? mR : mL;
    const double dB = dA - du;
    const double dK = takeL ? dA : dB, dO = takeL ? dB : dA;
    const double DK = suK - dK;
    const double iS = rcp_fast(SR - SL);
    const double bn = fma(SR, B.bn, -SL * A.bn) * iS;
    const double bbn = bn * bn;
    const double iK = rcp_fast(DK);
    const double rK = mK * iK;
    double isK, sK;
    rsqrt_and_sqrt(rK, isK, sK);
    const bool bnz = mag_ge(bn, kMag1em6 + 1);
    const double SA = bnz ? fma(takeL ? -dabs(bn) : dabs(bn), isK, SM) : SM;  // Alfven speed
    int level;
    if (takeL) level = ge_zero(SL) ? 0 : (ge_zero(SA) ? 1 : 2);
    else level = gt_zero(SA) ? 2 : (gt_zero(SR) ? 1 : 0);
    const double vsq = fma(Kun, Kun, Kut * Kut);
    const double KE = fma(Kp, P.inv_gm1, 0.5 * fma(Kr, vsq, Kbb));
    const double wKf = fma(Kun, Kbn, Kut * Kbt);

    // ---- reverse ------------------------------------------------------------------------
    const double Fm = Fb[0], Fmn = Fb[1], Fmt = Fb[2], Fe = Fb[3], Fbn = Fb[4], Fbt = Fb[5],
                 Fbz = Fb[6];
    SideB k = {}, o = {};
    double KEb, wKfb;               // adjoints of K's energy and of its u.b
    double SKb = 0.0, SOb = 0.0;    // of the two outer speeds
    if (level == 0) {
        // F0 = r un ; F1 = F0 un + pT - bn^2 ; F2 = F0 ut - bn bt ; F5 = un bt - ut bn ;
        // F6 = un bz ; F3 = (E + pT) un - bn (ut bt + un bn)
        const double F0 = Kr * Kun;
        const double F0b = fma(Fmt, Kut, fma(Fmn, Kun, Fm));
        KEb = Fe * Kun;
        wKfb = -Fe * Kbn;
        k.r = F0b * Kun;
        k.un = fma(F0b, Kr, fma(Fmn, F0, fma(Fbt, Kbt, fma(Fbz, Kbz, Fe * (KE + KpT)))));
        k.ut = fma(Fmt, F0, -Fbt * Kbn);
        k.pT = Fmn + KEb;
        k.bn = -fma(2.0 * Fmn, Kbn, fma(Fmt, Kbt, fma(Fbt, Kut, Fe * wKf)));
        k.bt = fma(Fbt, Kun, -Fmt * Kbn);
        k.bz = Fbz * Kun;
    } else {
        const StarV sk = star_fwd(mK, DK, dK, bn, bbn, Kut, Kbt, Kbz);
        const double PT = fma(mK, dK, KpT);
        const double phi = rK * SM;
        const double SMbn = SM * bn;
        const double sbK = fma(sk.w, sk.z, fma(sk.v, sk.b, SMbn));
        const double wsb = wKf - sbK;
        const double eK = fma(bn, wsb, fma(KE, suK, fma(PT, SM, -KpT * Kun))) * iK;
        // X: the double star at level 2, else K's star state
        double Xv = sk.v, Xw = sk.w, Xb = sk.b, Xz = sk.z, Xsb = sbK, Xe = eK;
        StarV so;
        double DO = 0, iO = 0, rO = 0, isO = 0, sO = 0, is = 0, dv = 0, dw = 0, v3 = 0, w3 = 0;
        // sign(bn) towards O
        const int sg = bnz ? ((gt_zero(bn) == takeL) ? 1 : -1) : 0;
        if (level == 2) {
            DO = suO - dO;
            iO = rcp_fast(DO);
            rO = mO * iO;
            rsqrt_and_sqrt(rO, isO, sO);
            so = star_fwd(mO, DO, dO, bn, bbn, Out, Obt, Obz);
            is = rcp_fast(sK + sO);
            dv = so.v - sk.v;
            dw = so.w - sk.w;
            v3 = fma(sO, dv, sgn_select(so.b - sk.b, sg)) * is;  // from K's star state
            w3 = fma(sO, dw, sgn_select(so.z - sk.z, sg)) * is;
            const double ss = sgn_select(sK, sg);
            Xv = sk.v + v3;
            Xw = sk.w + w3;
            Xb = fma(ss, v3, sk.b);
            Xz = fma(ss, w3, sk.z);
            Xsb = fma(Xw, Xz, fma(Xv, Xb, SMbn));
            Xe = fma(ss, Xsb - sbK, eK);
        }
        const double eb = Fe * SM;
        const double dbn = bn - Kbn;
        const double t0 = fma(Fmt, Kbt, fma(Fbt, Kut, Fe * wKf));
        double SMb = fma(phi, Fmn, fma(Xb, Fbt, fma(Xz, Fbz, Fe * (Xe + PT))));
        double PTb = Fmn + eb;
        double bnb = t0 - fma(Xb, Fmt, fma(Xv, Fbt, fma(Xw, Fbz, Xsb * Fe)));
        double vb = fma(phi, Fmt, -bn * Fbt), wb = -bn * Fbz;
        double bb = fma(SM, Fbt, -bn * Fmt), zb = SM * Fbz;
        double sbb = -bn * Fe;
        double rKb = fma(Fmn, SM, fma(Fmt, Xv, Fm));  // of phi
        SMb = fma(rKb, rK, SMb);
        rKb *= SM;
        wKfb = dbn * Fe;
        k.bn = -fma(2.0 * Fmn, Kbn, t0);
        k.bt = dbn * Fmt;
        k.ut = dbn * Fbt;
        double mKb = 0.0, mOb = 0.0, suKb = 0.0;
        if (!sk.g) {
            bnb = fma(-Fmt, Kbt, bnb);
            k.bt -= fma(Fmt, bn, Fbt * suK);
            k.bz = -Fbz * suK;
            suKb = -fma(Fbt, Kbt, Fbz * Kbz);
        }
        if (level == 2) {
            // e3 = eK + sg sK (sb3 - sbK), sb3 = w3 z3 + v3 b3 + SM bn
            const double t = sgn_select(eb, sg);
            double sKb = t * (Xsb - sbK);
            sbb = fma(t, sK, sbb);
            wb = fma(sbb, Xz, wb);
            zb = fma(sbb, Xw, zb);
            vb = fma(sbb, Xb, vb);
            bb = fma(sbb, Xv, bb);
            SMb = fma(sbb, bn, SMb);
            bnb = fma(sbb, SM, bnb);
            sbb = -t * sK;
            // (sK + sO) v3 = sK vK + sO vO + sg (bO - bK), b3 = bK + sg sK (v3 - vK): with
            // al = (v - sO sg b) / (sK + sO), be = (v + sK sg b) / (sK + sO) of the adjoints,
            // sK += (vK - v3) al, sO += (vO - v3) be, vK = sK al, vO = sO be, bK = -sg al,
            // bO = sg be; the same for w, z
            vb *= is;
            wb *= is;
            bb = sgn_select(bb, sg) * is;
            zb = sgn_select(zb, sg) * is;
            const double av = fma(-sO, bb, vb), bv = fma(sK, bb, vb);
            const double aw = fma(-sO, zb, wb), bw = fma(sK, zb, wb);
            sKb = fma(-v3, av, fma(-w3, aw, sKb));
            const double sOb = fma(dv - v3, bv, (dw - w3) * bw);
            vb = sK * av;
            wb = sK * aw;
            bb = sgn_select(av, -sg);
            zb = sgn_select(aw, -sg);
            // s = sqrt(r*): ds = 0.5 / s dr ; r* = m / D
            rKb = fma(0.5 * sKb, isK, rKb);
            mOb = 0.5 * sOb * isO * iO;
            double DOb = -mOb * rO, dOb = 0.0;
            star_rev(so, mO, DO, bn, Obt, Obz, sO * bv, sO * bw, sgn_select(bv, sg),
                     sgn_select(bw, sg), o, mOb, DOb, dOb, bnb);
            SOb = DOb;
            SMb += dOb - DOb;
            o.un = -dOb;
        }
        // D eK = E su + P* SM - pT un + bn (wKf - sbK)
        const double nb = eb * iK;
        KEb = nb * suK;
        suKb = fma(nb, KE, suKb);
        PTb = fma(nb, SM, PTb);
        SMb = fma(nb, PT, SMb);
        bnb = fma(nb, wsb, bnb);
        const double nbn = nb * bn;
        wKfb += nbn;
        sbb -= nbn;
        double DKb = -nb * eK, dKb = 0.0;
        // sbK = wK zK + vK bK + SM bn
        wb = fma(sbb, sk.z, wb);
        zb = fma(sbb, sk.w, zb);
        vb = fma(sbb, sk.b, vb);
        bb = fma(sbb, sk.v, bb);
        SMb = fma(sbb, bn, SMb);
        bnb = fma(sbb, SM, bnb);
        // rK = m / D ; the star state ; P* = pT + m d
        mKb = rKb * iK;
        DKb = fma(-mKb, rK, DKb);
        star_rev(sk, mK, DK, bn, Kbt, Kbz, vb, wb, bb, zb, k, mKb, DKb, dKb, bnb);
        mKb = fma(PTb, dK, mKb);
        dKb = fma(PTb, mK, dKb);
        SKb = DKb;
        SMb += dKb - DKb;
        // mR (SM - uR) + pR = mL (SM - uL) + pL
        const double ns = SMb * iden;
        const double nK = takeL ? -ns : ns;
        mKb = fma(-nK, dK, mKb);
        mOb = fma(nK, dO, mOb);
        // m = r su, su = S - un
        suKb = fma(mKb, Kr, suKb);
        const double suOb = mOb * Or;
        k.r = mKb * suK;
        o.r = mOb * suO;
        k.un = fma(nK, mK, -fma(nb, KpT, dKb)) - suKb;
        o.un = fma(-nK, mO, o.un) - suOb;
        k.pT = PTb - fma(nb, Kun, nK);
        o.pT = nK;
        SKb += suKb;
        SOb += suOb;
        // (SR - SL) bn = SR bR - SL bL
        const double nn = bnb * iS;
        const double nB = takeL ? -nn : nn;
        SKb = fma(nB, Kbn - bn, SKb);
        SOb = fma(-nB, Obn - bn, SOb);
        k.bn = fma(nB, SK, k.bn);
        o.bn = -nB * SO;
    }
    // E = p inv_gm1 + 0.5 (r (un^2 + ut^2) + bb) ; wKf = un bn + ut bt
    const double kin = 0.5 * KEb, rE = Kr * KEb;
    k.p = KEb * P.inv_gm1;
    k.bb = kin;
    k.r = fma(kin, vsq, k.r);
    k.un = fma(wKfb, Kbn, fma(rE, Kun, k.un));
    k.ut = fma(wKfb, Kbt, fma(rE, Kut, k.ut));
    k.bn = fma(wKfb, Kun, k.bn);
    k.bt = fma(wKfb, Kut, k.bt);
    // F.bn = -UU (B.bn - A.bn), UU = max(|SL|, |SR|)
    const double UU = dabs(UUR ? SR : SL);
    const double UUb = -Fbn * (B.bn - A.bn);
    double SLb = takeL ? SKb : SOb, SRb = takeL ? SOb : SKb;
    {
        add_to(UUR, SRb, SLb, sgn_select(UUb, lt_zero(UUR ? SR : SL) ? -1 : 1));
    }
    // back to A and B
    SideB Ab, Bb;
    Ab.r = takeL ? k.r : o.r;      Bb.r = takeL ? o.r : k.r;
    Ab.p = takeL ? k.p : 0.0;      Bb.p = takeL ? 0.0 : k.p;
    Ab.un = takeL ? k.un : o.un;   Bb.un = takeL ? o.un : k.un;
    Ab.ut = takeL ? k.ut : o.ut;   Bb.ut = takeL ? o.ut : k.ut;
    Ab.bn = takeL ? k.bn : o.bn;   Bb.bn = takeL ? o.bn : k.bn;
    Ab.bt = takeL ? k.bt : o.bt;   Bb.bt = takeL ? o.bt : k.bt;
    Ab.bz = takeL ? k.bz : o.bz;   Bb.bz = takeL ? o.bz : k.bz;
    Ab.pT = takeL ? k.pT : o.pT;   Bb.pT = takeL ? o.pT : k.pT;
    Ab.bb = takeL ? k.bb : 0.0;    Bb.bb = takeL ? 0.0 : k.bb;
    Ab.bn = fma(Fbn, UU, Ab.bn);
    Bb.bn = fma(-Fbn, UU, Bb.bn);
    // SL = uminN - cmax ; SR = umaxN + cmax
    const double cmaxb = SRb - SLb;
    add_to(minA, Ab.un, Bb.un, SLb);
    add_to(!maxB, Ab.un, Bb.un, SRb);
    // ---- the fast speed of the side of max(cf) ------------------------------------------
    {
        const double Ccf = cfB ? B.cf : A.cf, Crs = cfB ? B.rs : A.rs;
        const double Crq = cfB ? B.rq : A.rq, Ca = cfB ? B.a : A.a, Cgp = cfB ? B.gp : A.gp;
        const double Cbn2 = cfB ? B.bn2 : A.bn2, Cdisc = cfB ? B.disc : A.disc;
        // cf = X rsqrt(X r) = sqrt(X / r): d/dX = 0.5 rs, d/dr = -0.5 cf / r = -0.5 cf^2 rs
        const double Xh = 0.25 * cmaxb * Crs;  // half the adjoint of X
        const double rb = -2.0 * Xh * (Ccf * Ccf);
        // X = 0.5 (a + sq), sq = sqrt(disc), disc = a^2 - 4 gp bn2 (clamped at 0)
        double ab = Xh, gpb = 0.0, bn2b = 0.0;
        if ((bits(Cdisc) << 1) != 0) {
            const double sb = Xh * Crq;  // twice the adjoint of disc
            ab = fma(sb, Ca, ab);
            gpb = -2.0 * sb * Cbn2;
            bn2b = -2.0 * sb * Cgp;
        }
        gpb += ab;  // a = gp + bb
        add_to(!cfB, Ab.r, Bb.r, rb);
        add_to(!cfB, Ab.p, Bb.p, gpb * P.gamma);
        add_to(!cfB, Ab.bb, Bb.bb, ab);
        Ab.bn2 = cfB ? 0.0 : bn2b;
        Bb.bn2 = cfB ? bn2b : 0.0;
    }
    side_tail(A, Ab, qa_b);
    side_tail(B, Bb, qb_b);
}

// ---------------------------------------------------------------------------------------
// Pass B: face adjoints (each face once), then the gather into cells.
//
// B1 adj_face_kernel: one thread per face.  Bound by the FP64 pipe: 357 us for the 2 x 512^2
// faces of a 512^2 grid, 552 us when the sweep reversed the forward's chain of operations (512
// FP64 operations per face).  It reconstructs the face's two states from the
// four cells along its normal, recomputes the flux's star states and runs its reverse sweep on
// Fbar = k (dbar_low - dbar_high).  The adjoint of the low-side state (the upper face state
// of the low cell) goes to that cell's "up" plane, the adjoint of the high-side state (the
// lower face state of the high cell) to that cell's "dn" plane: every entry has exactly one
// writer.  The face thread also records, before its reverse sweep, the reconstruction
// choices of its two cells in bytes: for the low cell the minmod choice of its slope and
// whether its upper face state fell back to the cell value (rho, p), for the high cell
// whether its lower face state fell back (a fallback face state does not depend on the slope).
// Scratch layout after the 15 pass-A planes:
//   kFaceAdj + (dir * 2 + side) * 7 + f         face-state adjoints, side 0 = up, 1 = dn
//   kSel bytes, (dir * 7 + f) * K + cell        (choice + 1) | upper fallback << 2,
//                                               choice -1 left, +1 right, 0 none
//   kSel bytes, 14 K + (dir * 2 + f) * K + cell lower fallback (f < 2)
// dir 0 = x, 1 = y.
// B2 adj_gather_kernel: one thread per cell.  The cell's state adjoint collects the value
// parts of its two face states per direction, its own slope adjoint through its minmod
// choice, its neighbours' slope adjoints where their minmod choice used it, and the Powell
// terms of its neighbours, in a fixed order (deterministic).  Bound by the FP64 pipe: 52 us at
// 512^2, 69 us with the slope adjoints of all three cells formed before the choices.
// ---------------------------------------------------------------------------------------
constexpr int kFaceAdj = 15;
constexpr int kSel = kFaceAdj + 4 * NF;
constexpr int kScratchPlanes = kSel + 3;  // 18 bytes per cell fit in three planes of doubles
constexpr int FBX = 32, FBY = 4;  // 128-thread blocks of the gather
// B1: 64-thread blocks at five per SM (168 registers, 0.25 KB of spills per thread) took 5.90 ms
// for ten reverse steps on 512^2 cells; 5.95 ms without the bound (208 registers), 5.99 ms at
// six, 6.15 ms at eight per SM; 128-thread blocks 6.06 ms (208 registers), 5.99 ms at three per
// SM; 32-thread blocks 6.12 ms.
constexpr int kFaceRows = 2;

// periodic index for any i
__device__ __forceinline__ int wrap(int i, int n) {
    const int r = i % n;
    return r < 0 ? r + n : r;
}

// state value in b units (the field is stored in Gaussian units).  The product is rounded
// on its own (__dmul_rn: never fused into a later add), as the forward kernel rounds it when
// it stages the tile: equal neighbours then give an exact zero difference, and the minmod
// choices here are the forward's.
__device__ __forceinline__ double ld_b(const CPlanes& U, int f, long long k) {
    const double v = __ldg(U.f[f] + k);
    return f >= 4 ? __dmul_rn(v, kInvSpi4) : v;
}

// minmod slope and which difference it took: +1 right (c_{+1} - c), -1 left (c - c_{-1}), 0
__device__ __forceinline__ double slope_sel(double cm, double c, double cp, int& sel) {
    const double l = c - cm, r = cp - c;
    const double s = minmod(l, r);
    sel = mag(s) == 0 ? 0 : (mag_lt(r, l) ? 1 : -1);
    return s;
}

__global__ void __launch_bounds__(FBX * kFaceRows, 5) adj_face_kernel(
    Params P, CPlanes U, double* scratch, const double* __restrict__ T_do_ptr) {
    const int N = P.N, M = P.M;
    const long long K = (long long)N * M;
    const bool isx = blockIdx.y == 0;
    // blocks of a row first, then rows, in one grid dimension (the second one is too short)
    const unsigned nbx = (unsigned)((N + FBX - 1) / FBX);
    const int ix = (int)(blockIdx.x % nbx) * FBX + threadIdx.x;         // x-face index or column
    const int iy = (int)(blockIdx.x / nbx) * kFaceRows + threadIdx.y;  // row or y-face index
    if (ix >= N || iy >= M) return;
    const double T_do = *T_do_ptr;
    const double kk = T_do * (isx ? P.inv_dx : P.inv_dy);  // the forward's scaling
    // the face lies between cells a-1 and a along its normal; cells a-2 .. a+1
    long long kc[4];
#pragma unroll
    for (int t = 0; t < 4; ++t)
        kc[t] = isx ? (long long)iy * N + wrap(ix - 2 + t, N)
                    : (long long)wrap(iy - 2 + t, M) * N + ix;
    double c[4][NF];
#pragma unroll
    for (int t = 0; t < 4; ++t)
#pragma unroll
        for (int f = 0; f < NF; ++f) c[t][f] = ld_b(U, f, kc[t]);
    // face states: low cell (t=1) + its slope / 2, high cell (t=2) - its slope / 2
    double qa[NF], qb[NF];
    unsigned char* rec = reinterpret_cast<unsigned char*>(scratch + (size_t)kSel * K);
    unsigned char* sel = rec + (size_t)(isx ? 0 : NF) * K;
    unsigned char* fbl = rec + (size_t)(2 * NF + (isx ? 0 : 2)) * K;
#pragma unroll
    for (int f = 0; f < NF; ++f) {
        int sa, sb_;
        const double da = slope_sel(c[0][f], c[1][f], c[2][f], sa);
        const double db = slope_sel(c[1][f], c[2][f], c[3][f], sb_);
        const double va = fma(0.5, da, c[1][f]), vb = fma(-0.5, db, c[2][f]);
        const bool fu = f < 2 && le_zero(va), fd = f < 2 && le_zero(vb);
        qa[f] = fu ? c[1][f] : va;
        qb[f] = fd ? c[2][f] : vb;
        sel[(size_t)f * K + kc[1]] = (unsigned char)((sa + 1) | (fu ? 4 : 0));  // low cell
        if (f < 2) fbl[(size_t)f * K + kc[2]] = fd ? 1 : 0;                   // high cell
    }
    // flux adjoint: d_low += k F, d_high -= k F
    double Fslot[NF];
#pragma unroll
    for (int f = 0; f < NF; ++f)
        Fslot[f] = kk * (scratch[(size_t)(7 + f) * K + kc[1]] - scratch[(size_t)(7 + f) * K + kc[2]]);
    // slots: 0 m, 1 e, 2 mx, 3 my, 4 bx, 5 by, 6 bz -> local (m, mn, mt, e, bn, bt, bz)
    const double Fb[7] = {Fslot[0], isx ? Fslot[2] : Fslot[3], isx ? Fslot[3] : Fslot[2],
                          Fslot[1], isx ? Fslot[4] : Fslot[5], isx ? Fslot[5] : Fslot[4],
                          Fslot[6]};
    const double la[7] = {qa[0], qa[1], isx ? qa[2] : qa[3], isx ? qa[3] : qa[2],
                          isx ? qa[4] : qa[5], isx ? qa[5] : qa[4], qa[6]};
    const double lb[7] = {qb[0], qb[1], isx ? qb[2] : qb[3], isx ? qb[3] : qb[2],
                          isx ? qb[4] : qb[5], isx ? qb[5] : qb[4], qb[6]};
    double lab[7], lbb[7];
    hlld_vjp(la, lb, Fb, P, lab, lbb);
    // back to field order (rho, p, vx, vy, bx, by, bz)
    const double gab[7] = {lab[0], lab[1], isx ? lab[2] : lab[3], isx ? lab[3] : lab[2],
                           isx ? lab[4] : lab[5], isx ? lab[5] : lab[4], lab[6]};
    const double gbb[7] = {lbb[0], lbb[1], isx ? lbb[2] : lbb[3], isx ? lbb[3] : lbb[2],
                           isx ? lbb[4] : lbb[5], isx ? lbb[5] : lbb[4], lbb[6]};
    double* up = scratch + (size_t)(kFaceAdj + (isx ? 0 : 2) * NF) * K;
    double* dn = up + (size_t)NF * K;
#pragma unroll
    for (int f = 0; f < NF; ++f) {
        up[(size_t)f * K + kc[1]] = gab[f];
        dn[(size_t)f * K + kc[2]] = gbb[f];
    }
}

__global__ void __launch_bounds__(FBX * FBY) adj_gather_kernel(Params P,
                                                               const double* __restrict__ scratch,
                                                               Planes lam_in,
                                                               const double* __restrict__ T_do_ptr) {
    const int N = P.N, M = P.M;
    const long long K = (long long)N * M;
    const int gx = blockIdx.x * FBX + threadIdx.x, gy = blockIdx.y * FBY + threadIdx.y;
    if (gx >= N || gy >= M) return;
    const long long k = (long long)gy * N + gx;
    const double T_do = *T_do_ptr;
    const double kx = T_do * P.inv_dx, ky = T_do * P.inv_dy;
    double lam[NF];
#pragma unroll
    for (int f = 0; f < NF; ++f) lam[f] = scratch[(size_t)f * K + k];
    const unsigned char* rec = reinterpret_cast<const unsigned char*>(scratch + (size_t)kSel * K);
#pragma unroll
    for (int dir = 0; dir < 2; ++dir) {
        const bool isx = dir == 0;
        // the cells at positions -1, 0, +1 along the direction
        long long kc[3];
#pragma unroll
        for (int t = 0; t < 3; ++t)
            kc[t] = isx ? (long long)gy * N + wrap(gx - 1 + t, N)
                        : (long long)wrap(gy - 1 + t, M) * N + gx;
        const double* up = scratch + (size_t)(kFaceAdj + 2 * dir * NF) * K;
        const double* dn = up + (size_t)NF * K;
        const unsigned char* sel = rec + (size_t)dir * NF * K;
        const unsigned char* fbl = rec + (size_t)(2 * NF + 2 * dir) * K;
#pragma unroll
        for (int f = 0; f < NF; ++f) {
            const double* upf = up + (size_t)f * K;
            const double* dnf = dn + (size_t)f * K;
            int s[3];
            bool fu[3], fd[3];
#pragma unroll
            for (int t = 0; t < 3; ++t) {
                const int b = sel[(size_t)f * K + kc[t]];
                s[t] = (b & 3) - 1;
                fu[t] = (b & 4) != 0;
                fd[t] = f < 2 && fbl[(size_t)f * K + kc[t]] != 0;
            }
            // The slope adjoint of a cell is half of up - dn, a fallback face state dropping its
            // term.  Value parts and the cell's own slope (left difference c - c_{-1} -> +1,
            // right one -> -1): up (1 +- 1/2) + dn (1 -+ 1/2).
            double acc = fma(fu[1] || s[1] == 0 ? 1.0 : (s[1] == -1 ? 1.5 : 0.5), upf[k], lam[f]);
            acc = fma(fd[1] || s[1] == 0 ? 1.0 : (s[1] == -1 ? 0.5 : 1.5), dnf[k], acc);
            // neighbour -1 took its right difference (c - c_{-1}); neighbour +1 its left one
            const bool a = s[0] == 1, c = s[2] == -1;
            const double x = (a && !fu[0] ? upf[kc[0]] : 0.0) - (a && !fd[0] ? dnf[kc[0]] : 0.0);
            const double y = (c && !fu[2] ? upf[kc[2]] : 0.0) - (c && !fd[2] ? dnf[kc[2]] : 0.0);
            lam[f] = fma(0.5, x - y, acc);
        }
    }
    // Powell: divb_c' = 0.5 kx (bx_{c'+1} - bx_{c'-1}) + 0.5 ky (by_{c'+N} - by_{c'-N})
    {
        const long long kW = (long long)gy * N + wrap(gx - 1, N);
        const long long kE = (long long)gy * N + wrap(gx + 1, N);
        const long long kS = (long long)wrap(gy - 1, M) * N + gx;
        const long long kN = (long long)wrap(gy + 1, M) * N + gx;
        const double* dvb = scratch + (size_t)14 * K;
        lam[4] += 0.5 * kx * (dvb[kW] - dvb[kE]);
        lam[5] += 0.5 * ky * (dvb[kS] - dvb[kN]);
    }
    // field adjoint back to the stored Gaussian units: b = B / sqrt(4 pi)
    lam[4] *= kInvSpi4;
    lam[5] *= kInvSpi4;
    lam[6] *= kInvSpi4;
#pragma unroll
    for (int f = 0; f < NF; ++f) lam_in.f[f][k] = lam[f];
}

int grid_cells(long long K) {
    long long g = (K + NT - 1) / NT;
    return (int)(g > 152 * 16 ? 152 * 16 : (g < 1 ? 1 : g));
}

// ---------------------------------------------------------------------------------------
// Branch switches between two runs (gd_adj_switches).  A central difference of runs from
// U0 + eps v and U0 - eps v is the derivative of the branch both take only where every
// non-smooth choice comes out the same in both.  Per face, the choices its flux depends on,
// computed from the FP64 quantities that adj_face_kernel takes its branches by: the minmod
// pick of its low cell's slope (every cell's slope is counted at exactly one face per
// direction), the rho / p fallbacks of its two face states, and the HLLD choices: which
// side gives min(u), max(u), max(cf) and max(|S|) (speeds), the upwind side and the region
// of the fan (region), and the guards disc <= 0, |tt| >= 1e-5 on both sides, |bn| > 1e-6
// and sign(bn) (guards).  Per cell, the update's floors rho <= 0 and p <= 0.  Counters
// (kSw*): (step, face) pairs per face category, (step, cell) pairs for floors and for
// cells touched by any switch, and, at the end, the cells switched at any step.
// ---------------------------------------------------------------------------------------
struct FaceCode {
    unsigned int minmod, fallback, speeds, region, guards;
};

__device__ __forceinline__ FaceCode face_code(const Params& P, const CPlanes& U, bool isx,
                                              const long long* kc) {
    FaceCode code{0u, 0u, 0u, 0u, 0u};
    double c[4][NF];
#pragma unroll
    for (int t = 0; t < 4; ++t)
#pragma unroll
        for (int f = 0; f < NF; ++f) c[t][f] = ld_b(U, f, kc[t]);
    double qa[NF], qb[NF];
#pragma unroll
    for (int f = 0; f < NF; ++f) {
        int sa, sb_;
        const double da = slope_sel(c[0][f], c[1][f], c[2][f], sa);
        const double db = slope_sel(c[1][f], c[2][f], c[3][f], sb_);
        const double va = fma(0.5, da, c[1][f]), vb = fma(-0.5, db, c[2][f]);
        const bool fu = f < 2 && le_zero(va), fd = f < 2 && le_zero(vb);
        qa[f] = fu ? c[1][f] : va;
        qb[f] = fd ? c[2][f] : vb;
        code.minmod |= (unsigned int)(sa + 1) << (2 * f);
        if (f < 2) code.fallback |= (fu ? 1u : 0u) << (2 * f) | (fd ? 2u : 0u) << (2 * f);
    }
    const double la[7] = {qa[0], qa[1], isx ? qa[2] : qa[3], isx ? qa[3] : qa[2],
                          isx ? qa[4] : qa[5], isx ? qa[5] : qa[4], qa[6]};
    const double lb[7] = {qb[0], qb[1], isx ? qb[2] : qb[3], isx ? qb[3] : qb[2],
                          isx ? qb[4] : qb[5], isx ? qb[5] : qb[4], qb[6]};
    SideV A, B;
    side_fwd(A, la, P);
    side_fwd(B, lb, P);
    // the forward part of hlld_vjp up to the region, for both sides
    const bool minA = !dlt(B.un, A.un);
    const bool maxB = dlt(A.un, B.un);
    const double uminN = minA ? A.un : B.un;
    const double umaxN = maxB ? B.un : A.un;
    const bool cfB = mag_lt(A.cf, B.cf);
    const double cmax = cfB ? B.cf : A.cf;
    const double SL = uminN - cmax, SR = umaxN + cmax;
    const double suL = SL - A.un, suR = SR - B.un;
    const double mL = A.r * suL, mR = B.r * suR;
    const double iden = rcp_fast(mR - mL);
    const double SM = A.un + fma(mR, B.un - A.un, A.pT - B.pT) * iden;
    const bool UUR = mag_lt(SL, SR);
    const double iS = rcp_fast(SR - SL);
    const double bn = fma(SR, B.bn, -SL * A.bn) * iS;
    const double iL = rcp_fast(SL - SM), iR = rcp_fast(SR - SM);
    const double rLL = mL * iL, rRR = mR * iR;
    const double bbn = bn * bn;
    const double ttL = fma(mL, SL - SM, -bbn);
    const bool gL = mag_ge(ttL, kMag1em5);
    const double ttR = fma(mR, SR - SM, -bbn);
    const bool gR = mag_ge(ttR, kMag1em5);
    double isLL, isRR, sLL, sRR;
    rsqrt_and_sqrt(rLL, isLL, sLL);
    rsqrt_and_sqrt(rRR, isRR, sRR);
    const bool bnz = mag_ge(bn, kMag1em6 + 1);
    const double abn = dabs(bn);
    const double SLL = bnz ? fma(-abn, isLL, SM) : SM;
    const double SRR = bnz ? fma(abn, isRR, SM) : SM;
    const bool takeL = ge_zero(SL) || ge_zero(SM);
    int level;
    if (takeL) level = ge_zero(SL) ? 0 : (ge_zero(SLL) ? 1 : 2);
    else level = gt_zero(SRR) ? 2 : (gt_zero(SR) ? 1 : 0);
    code.speeds = (minA ? 1u : 0u) | (maxB ? 2u : 0u) | (cfB ? 4u : 0u) | (UUR ? 8u : 0u);
    code.region = (takeL ? 1u : 0u) | ((unsigned int)level << 1);
    code.guards = (A.disc0 ? 1u : 0u) | (B.disc0 ? 2u : 0u) | (gL ? 4u : 0u) | (gR ? 8u : 0u) |
                  (bnz ? 16u : 0u) | (bnz && lt_zero(bn) ? 32u : 0u);
    return code;
}

// warp-aggregated counter increment: one atomic per warp and kind
__device__ __forceinline__ void count_if(unsigned long long* ctr, bool hit) {
    const unsigned int m = __ballot_sync(0xffffffffu, hit);
    if (m != 0u && (threadIdx.x & 31) == (unsigned)(__ffs((int)m) - 1))
        atomicAdd(ctr, (unsigned long long)__popc(m));
}

__global__ void __launch_bounds__(FBX * FBY) switch_face_kernel(Params P, CPlanes Ua, CPlanes Ub,
                                                                unsigned long long* ctr,
                                                                unsigned char* step_mark) {
    const int N = P.N, M = P.M;
    const bool isx = blockIdx.z == 0;
    const int ix = blockIdx.x * FBX + threadIdx.x;
    const int iy = blockIdx.y * FBY + threadIdx.y;
    const bool in = ix < N && iy < M;
    FaceCode a{0u, 0u, 0u, 0u, 0u}, b{0u, 0u, 0u, 0u, 0u};
    long long kc[4] = {0, 0, 0, 0};
    if (in) {
#pragma unroll
        for (int t = 0; t < 4; ++t)
            kc[t] = isx ? (long long)iy * N + wrap(ix - 2 + t, N)
                        : (long long)wrap(iy - 2 + t, M) * N + ix;
        a = face_code(P, Ua, isx, kc);
        b = face_code(P, Ub, isx, kc);
    }
    const bool sm = a.minmod != b.minmod, sf = a.fallback != b.fallback;
    const bool ss = a.speeds != b.speeds, sr = a.region != b.region, sg = a.guards != b.guards;
    // counted per warp: threadIdx is 32 x 4, so each warp is one threadIdx.y row
    count_if(ctr + 0, sm);
    count_if(ctr + 1, sf);
    count_if(ctr + 2, ss);
    count_if(ctr + 3, sr);
    count_if(ctr + 4, sg);
    if (sm || sf || ss || sr || sg) {
        // the slope of the low cell, both face states and the flux between them
        step_mark[kc[1]] = 1;
        step_mark[kc[2]] = 1;
    }
}

// Floors of the update of U (with the forward's flux differences and Powell term aux), as
// adj_update_kernel recomputes them: bit 0 rho <= 0, bit 1 p <= 0.
__device__ __forceinline__ unsigned int floor_code(const Params& P, const CPlanes& U,
                                                   const double* aux, long long K, long long k) {
    const double r = U.f[0][k], p = U.f[1][k], u = U.f[2][k], v = U.f[3][k];
    const double bx = __dmul_rn(U.f[4][k], kInvSpi4), by = __dmul_rn(U.f[5][k], kInvSpi4);
    const double bz = __dmul_rn(U.f[6][k], kInvSpi4);
    double d[NF];
#pragma unroll
    for (int f = 0; f < NF; ++f) d[f] = aux[(size_t)f * K + k];
    const double divb = aux[(size_t)7 * K + k];
    const double ub = fma(u, bx, v * by);
    const double bb = fma(bz, bz, fma(by, by, bx * bx));
    const double K1 = fma(r, fma(u, u, v * v), bb);
    double r2 = r - d[0];
    const bool rfl = le_zero(r2);
    if (rfl) r2 = r;
    const double mx2 = fma(r, u, -fma(bx, divb, d[2]));
    const double my2 = fma(r, v, -fma(by, divb, d[3]));
    const double bx2 = bx - fma(u, divb, d[4]);
    const double by2 = by - fma(v, divb, d[5]);
    const double bz2 = bz - d[6];
    const double dE = fma(ub, divb, d[1]);
    const double inv = rcp_fast(r2);
    const double u2 = mx2 * inv, v2 = my2 * inv;
    const double K2 = fma(r2, fma(u2, u2, v2 * v2), fma(bz2, bz2, fma(by2, by2, bx2 * bx2)));
    const double p2 = fma(P.hgm1, K1 - K2, fma(-P.gm1, dE, p));
    return (rfl ? 1u : 0u) | (le_zero(p2) ? 2u : 0u);
}

__global__ void __launch_bounds__(NT) switch_cell_kernel(Params P, CPlanes Ua, const double* auxa,
                                                         CPlanes Ub, const double* auxb,
                                                         unsigned long long* ctr,
                                                         unsigned char* step_mark,
                                                         unsigned char* ever_mark) {
    const long long K = (long long)P.N * P.M;
    const long long stride = (long long)gridDim.x * blockDim.x;
    const long long K_up = (K + 31) / 32 * 32;  // whole warps through the loop (ballots)
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < K_up; k += stride) {
        bool fl = false, any = false;
        if (k < K) {
            fl = floor_code(P, Ua, auxa, K, k) != floor_code(P, Ub, auxb, K, k);
            any = fl || step_mark[k] != 0;
            if (any) {
                ever_mark[k] = 1;
                step_mark[k] = 0;
            }
        }
        count_if(ctr + 5, fl);
        count_if(ctr + 6, any);
    }
}

__global__ void __launch_bounds__(NT) switch_total_kernel(long long K,
                                                          const unsigned char* ever_mark,
                                                          unsigned long long* ctr) {
    const long long stride = (long long)gridDim.x * blockDim.x;
    const long long K_up = (K + 31) / 32 * 32;
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < K_up; k += stride)
        count_if(ctr + 7, k < K && ever_mark[k] != 0);
}

}  // namespace

int switch_kinds() { return 8; }

cudaError_t launch_switch_faces(const Params& P, const CPlanes& Ua, const CPlanes& Ub,
                                unsigned long long* ctr, unsigned char* step_mark,
                                cudaStream_t st) {
    const unsigned gxb = (unsigned)((P.N + FBX - 1) / FBX), gyb = (unsigned)((P.M + FBY - 1) / FBY);
    if (gyb > 65535u) return cudaErrorInvalidConfiguration;
    switch_face_kernel<<<dim3(gxb, gyb, 2), dim3(FBX, FBY), 0, st>>>(P, Ua, Ub, ctr, step_mark);
    return cudaGetLastError();
}

cudaError_t launch_switch_cells(const Params& P, const CPlanes& Ua, const double* auxa,
                                const CPlanes& Ub, const double* auxb, unsigned long long* ctr,
                                unsigned char* step_mark, unsigned char* ever_mark,
                                cudaStream_t st) {
    const long long K = (long long)P.N * P.M;
    switch_cell_kernel<<<grid_cells(K), NT, 0, st>>>(P, Ua, auxa, Ub, auxb, ctr, step_mark,
                                                     ever_mark);
    return cudaGetLastError();
}

cudaError_t launch_switch_total(long long K, const unsigned char* ever_mark,
                                unsigned long long* ctr, cudaStream_t st) {
    switch_total_kernel<<<grid_cells(K), NT, 0, st>>>(K, ever_mark, ctr);
    return cudaGetLastError();
}

int adjoint_scratch_planes() { return kScratchPlanes; }

cudaError_t prepare_adjoint() { return cudaSuccess; }

cudaError_t launch_adjoint_step(const Params& P, const CPlanes& U, const double* aux,
                                const CPlanes& lam_out, const Planes& lam_in, double* scratch,
                                const double* T_do, cudaStream_t st) {
    const long long K = (long long)P.N * P.M;
    const dim3 blk(FBX, FBY);
    const unsigned gxb = (unsigned)((P.N + FBX - 1) / FBX), gyb = (unsigned)((P.M + FBY - 1) / FBY);
    if (gyb > 65535u) return cudaErrorInvalidConfiguration;
    adj_update_kernel<<<grid_cells(K), NT, 0, st>>>(P, U, aux, lam_out, scratch);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    const unsigned fyb = (unsigned)((P.M + kFaceRows - 1) / kFaceRows);
    adj_face_kernel<<<dim3(gxb * fyb, 2), dim3(FBX, kFaceRows), 0, st>>>(P, U, scratch, T_do);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    adj_gather_kernel<<<dim3(gxb, gyb, 1), blk, 0, st>>>(P, scratch, lam_in, T_do);
    return cudaGetLastError();
}

}  // namespace gd
