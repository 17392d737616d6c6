// Host check of the face solvers in scaled 64-bit integers (gd_fixed.cuh, gd_fixed_mhd.cuh)
// against the same fluxes written out in long double.  Usage: fixed_check <faces per class>.
// One line per solver and class: the faces the integer solver took, those it left to the
// floating-point one, and the largest difference of a flux component or of the fan speed, over
// the larger side's scale of that component (density x fan speed^k, field x fan speed).
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

#include "../golikov_2d_gb300/csrc/gd_fixed_mhd.cuh"

using namespace gd;
using L = long double;

// state (r, p, un, ut, bn, bt, bz) of side i, conserved (r, mn, mt, e, -, bt, bz) and flux
struct Side {
    L r, p, u, v, n, t, z, bb, pt, E, ub, U[7], F[7];
};

static Side side(const double* q, bool mhd, L g) {
    Side s{};
    s.r = q[0]; s.p = q[1]; s.u = q[2]; s.v = q[3];
    if (mhd) { s.n = q[4]; s.t = q[5]; s.z = q[6]; }
    s.bb = s.n * s.n + s.t * s.t + s.z * s.z;
    s.pt = s.p + s.bb / 2;
    s.E = s.p / (g - 1) + s.r * (s.u * s.u + s.v * s.v) / 2 + s.bb / 2;
    s.ub = s.u * s.n + s.v * s.t;
    const L U[7] = {s.r, s.r * s.u, s.r * s.v, s.E, 0, s.t, s.z};
    const L F[7] = {s.r * s.u, s.r * s.u * s.u + s.pt - s.n * s.n, s.r * s.u * s.v - s.n * s.t,
                    (s.E + s.pt) * s.u - s.n * s.ub, 0, s.u * s.t - s.v * s.n, s.u * s.z};
    for (int k = 0; k < 7; ++k) { s.U[k] = U[k]; s.F[k] = F[k]; }
    return s;
}

enum Solver { HLLC, HLL, HLLD, HLLC_MHD };

// F[0..6] as in Side::F (F[4]: the diffusive normal-field flux), F[7]: max(|SL|, |SR|)
static void flux(Solver m, const double* qa, const double* qb, L g, L* F) {
    const bool mhd = m == HLLD || m == HLLC_MHD;
    const Side s[2] = {side(qa, mhd, g), side(qb, mhd, g)};
    L c[2];
    for (int i = 0; i < 2; ++i) {
        const L a = g * s[i].p + s[i].bb, d = a * a - 4 * g * s[i].p * s[i].n * s[i].n;
        c[i] = sqrtl((a + sqrtl(d < 0 ? 0 : d)) / (2 * s[i].r));
    }
    const L cm = fmaxl(c[0], c[1]);
    L S[2] = {fminl(s[0].u, s[1].u) - cm, fmaxl(s[0].u, s[1].u) + cm};
    if (m == HLLC) {  // the extreme sums of each side's own speed of sound
        S[0] = fminl(s[0].u - c[0], s[1].u - c[1]);
        S[1] = fmaxl(s[0].u + c[0], s[1].u + c[1]);
    }
    F[7] = fmaxl(-S[0], S[1]);
    if (m == HLL) {
        for (int k = 0; k < 7; ++k)
            F[k] = S[0] > 0 ? s[0].F[k] : S[1] < 0 ? s[1].F[k]
                 : (S[1] * s[0].F[k] - S[0] * s[1].F[k] + S[0] * S[1] * (s[1].U[k] - s[0].U[k])) /
                       (S[1] - S[0]);
        return;
    }
    L mm[2], su[2];
    for (int i = 0; i < 2; ++i) { su[i] = S[i] - s[i].u; mm[i] = s[i].r * su[i]; }
    const L SM = (mm[1] * s[1].u - mm[0] * s[0].u - s[1].pt + s[0].pt) / (mm[1] - mm[0]);
    const L PT = (mm[1] * s[0].pt - mm[0] * s[1].pt + mm[0] * mm[1] * (s[1].u - s[0].u)) /
                 (mm[1] - mm[0]);
    const L bn = (S[1] * s[1].n - S[0] * s[0].n) / (S[1] - S[0]);
    // star states: tangential velocity and field, energy
    L rs[2], v[2], w[2], b[2], z[2], sb[2], e[2], q[2];
    L hll[7], wz = 0;  // the fan's mean state (HLLC-MHD)
    for (int k = 0; k < 7; ++k)
        hll[k] = (S[1] * s[1].U[k] - S[0] * s[0].U[k] + s[0].F[k] - s[1].F[k]) / (S[1] - S[0]);
    wz = (s[1].n * s[1].z - s[0].n * s[0].z) / (S[1] - S[0]);
    for (int i = 0; i < 2; ++i) {
        rs[i] = mm[i] / (S[i] - SM);
        q[i] = sqrtl(rs[i]);
        const L tt = mm[i] * (S[i] - SM) - bn * bn;
        const bool ok = fabsl(tt) >= 1e-5L;
        v[i] = s[i].v; w[i] = 0; b[i] = 0; z[i] = 0;
        if (m == HLLC || m == HLLC_MHD) {
            if (m == HLLC_MHD) { v[i] = hll[2] / hll[0]; b[i] = hll[5]; z[i] = hll[6]; }
            sb[i] = m == HLLC ? 0 : (bn * hll[1] + hll[5] * hll[2] + hll[6] * wz) / hll[0];
        } else {
            if (ok) {
                const L k = bn * (SM - s[i].u) / tt, d = (mm[i] * su[i] - bn * bn) / tt;
                v[i] -= k * s[i].t; w[i] = -k * s[i].z; b[i] = d * s[i].t; z[i] = d * s[i].z;
            }
            sb[i] = SM * bn + v[i] * b[i] + w[i] * z[i];
        }
        e[i] = (s[i].E * su[i] + PT * SM - s[i].pt * s[i].u + bn * (s[i].ub - sb[i])) / (S[i] - SM);
    }
    const int i = S[0] >= 0 || SM >= 0 ? 0 : 1;
    const L sg = m != HLLD || fabsl(bn) <= 1e-6L ? 0 : bn > 0 ? 1 : -1;
    const L SA = SM + (i ? 1 : -1) * fabsl(sg * bn) / q[i];
    int level = i == 0 ? (S[0] >= 0 ? 0 : 1) : (S[1] > 0 ? 1 : 0);
    if (m == HLLD && level == 1 && (i == 0 ? SA < 0 : SA > 0)) level = 2;
    const L Us[7] = {rs[i], rs[i] * SM, rs[i] * v[i], e[i], 0, b[i], z[i]};
    const L Q = q[0] + q[1];
    const L v3 = (q[0] * v[0] + q[1] * v[1] + sg * (b[1] - b[0])) / Q;
    const L w3 = (q[0] * w[0] + q[1] * w[1] + sg * (z[1] - z[0])) / Q;
    const L b3 = (q[0] * b[1] + q[1] * b[0] + sg * q[0] * q[1] * (v[1] - v[0])) / Q;
    const L z3 = (q[0] * z[1] + q[1] * z[0] + sg * q[0] * q[1] * (w[1] - w[0])) / Q;
    const L e3 = e[i] + (i ? 1 : -1) * sg * q[i] * (sb[i] - (SM * bn + v3 * b3 + w3 * z3));
    const L U3[7] = {rs[i], rs[i] * SM, rs[i] * v3, e3, 0, b3, z3};
    for (int k = 0; k < 7; ++k) {
        F[k] = s[i].F[k];
        if (level >= 1) F[k] += S[i] * (Us[k] - s[i].U[k]);
        if (level == 2) F[k] += SA * (U3[k] - Us[k]);
    }
    F[4] = -F[7] * (s[1].n - s[0].n);
}

int main(int argc, char** argv) {
    const long n = argc > 1 ? atol(argv[1]) : 20000;
    std::mt19937_64 R(20260105);
    auto U = [&](double a, double b) { return a + (b - a) * (double)(R() >> 11) * 0x1p-53; };
    const char* solver[] = {"hllc", "hll", "hlld", "hllc_mhd"};
    // class: jump between the sides, Mach number, log range of the units, plasma beta
    struct { const char* name; double jump, mach, units, beta; } cls[] = {
        {"ordinary", 0.5, 0.7, 2, 1},       {"small_jumps", 1e-4, 0.7, 2, 1},
        {"tiny_jumps", 1e-9, 0.7, 2, 1},    {"slow", 0.3, 1e-4, 2, 1},
        {"supersonic", 0.3, 4, 2, 1},       {"strong_jumps", 1.2, 0.7, 2, 1},
        {"any_units", 0.3, 0.7, 40, 1},     {"strong_field", 0.3, 0.7, 2, 0.1},
        {"weak_field", 0.3, 0.7, 2, 1e6}};
    for (int m = 0; m < 4; ++m)
        for (const auto& c : cls) {
            const bool mhd = m >= HLLD;
            long taken = 0, left = 0;
            double worst = 0;
            for (long it = 0; it < n; ++it) {
                const double g = it & 1 ? 1.4 : it % 6 ? 5.0 / 3.0 : 1.1;
                const double r0 = exp(U(-c.units, c.units)), p0 = exp(U(-c.units, c.units));
                const double b0 = sqrt(p0 / c.beta), uc = sqrt(g * p0 / r0 + (mhd ? b0 * b0 / r0 : 0));
                const double u0 = uc * c.mach * U(-1, 1), v0 = uc * U(-1, 1);
                const double f0[3] = {b0 * U(-1, 1), b0 * U(-1, 1), b0 * U(-1, 1)};
                double q[14];
                for (int s = 0; s < 2; ++s) {
                    double* x = q + 7 * s;
                    x[0] = r0 * exp(c.jump * U(-1, 1));
                    x[1] = p0 * exp(c.jump * U(-1, 1));
                    x[2] = u0 + uc * c.jump * fmin(c.mach, 1) * U(-1, 1);
                    x[3] = v0 + uc * c.jump * U(-1, 1);
                    for (int k = 0; k < 3; ++k) x[4 + k] = f0[k] + b0 * c.jump * (k ? 1 : 0.1) * U(-1, 1);
                }
                // exact zeros and ties
                for (int s = 0; s < 2; ++s) {
                    double* x = q + 7 * s;
                    if (it % 41 == 0) x[2] = 0;
                    if (it % 43 == 0) x[3] = 0;
                    if (it % 47 == 0) x[4] = 0;
                    if (it % 53 == 0) x[4] = x[5] = x[6] = 0;
                    if (it % 59 == 0) for (int k = 0; k < 7; ++k) x[k] = q[k];
                }
                const fx::Gas G = fx::gas_of(g);
                double f[8] = {0, 0, 0, 0, 0, 0, 0, 0};
                bool ok;
                if (mhd) {
                    fx::FluxI o;
                    ok = m == HLLD ? fx::mhd_face<true>(q, q + 7, G, o, f[7])
                                   : fx::mhd_face<false>(q, q + 7, G, o, f[7]);
                    const double t[7] = {o.m, o.mn, o.mt, o.e, o.bn, o.bt, o.bz};
                    for (int k = 0; k < 7; ++k) f[k] = t[k];
                } else {
                    ok = m == HLLC ? fx::euler_face<false>(q, q + 7, G, f, f[7])
                                   : fx::euler_face<true>(q, q + 7, G, f, f[7]);
                    f[4] = 0;
                }
                if (!ok) { ++left; continue; }
                ++taken;
                L F[8];
                flux((Solver)m, q, q + 7, g, F);
                const double r = fmax(q[0], q[7]), S = (double)F[7];
                const double B = mhd ? fmax(b0, sqrt(r) * S * 1e-3) : 1.0;
                const double sc[8] = {r * S, r * S * S, r * S * fmax(S, fabs(v0)),
                                      r * S * fmax(S * S, v0 * v0), B * S, B * S, B * S, S};
                for (int k = 0; k < 8; ++k) {
                    const double d = fabs((double)((L)f[k] - F[k])) / sc[k];
                    if (!(d <= worst)) worst = d;
                }
            }
            printf("%s %s taken %ld left %ld worst %.3e\n", solver[m], c.name, taken, left, worst);
        }
}
