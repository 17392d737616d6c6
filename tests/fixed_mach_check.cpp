// Host check of the integer face solvers in fast flows: along the face, through it, and obliquely,
// at fast Mach numbers up to 1000, and through one side of it only.  Usage: fixed_mach_check <faces
// per class>.  One line per solver, class and Mach number: the faces taken and left, and the largest
// error of a flux component over its scale (with V the flow's speed beside the fan's S: transverse
// momentum density x S x V, energy density x S x V^2 with V >= S, transverse field S x field + V x
// normal field).
#define main ordinary_faces
#include "fixed_check.cpp"
#undef main

int main(int argc, char** argv) {
    const long n = argc > 1 ? atol(argv[1]) : 20000;
    std::mt19937_64 R(20260113);
    auto U = [&](double a, double b) { return a + (b - a) * (double)(R() >> 11) * 0x1p-53; };
    const char* solver[] = {"hllc", "hll", "hlld", "hllc_mhd"};
    struct { const char* name; double un, ut; bool one; } cls[] = {
        {"along", 0, 1, false}, {"through", 1, 0, false}, {"oblique", 1, 1, false},
        {"shallow", 0.1, 1, false}, {"one_side", 1, 0, true}};
    for (int m = 0; m < 4; ++m)
        for (const auto& c : cls)
            for (double mach : {2., 5., 8., 12., 20., 50., 1000.}) {
                const bool mhd = m >= HLLD;
                long taken = 0, left = 0;
                double worst = 0;
                for (long it = 0; it < n; ++it) {
                    const double g = it & 1 ? 1.4 : 5.0 / 3.0;
                    const double cs = std::sqrt(g * 0.7 + (mhd ? 1.0 : 0.0));  // r = 1, p = 0.7, |b| = 1
                    const double V = mach * cs * (it & 2 ? 1 : -1);
                    double q[14];
                    for (int s = 0; s < 2; ++s) {
                        double* x = q + 7 * s;
                        const double w = c.one && s == (it >> 2 & 1) ? 0 : 1;
                        x[0] = U(0.8, 1.25);
                        x[1] = 0.7 * U(0.8, 1.25);
                        x[2] = w * c.un * V + 0.4 * cs * U(-1, 1);
                        x[3] = w * c.ut * V + 0.4 * cs * U(-1, 1);
                        x[4] = 0.6 * U(-1, 1);
                        x[5] = 0.6 * U(-1, 1);
                        x[6] = 0.6 * U(-1, 1);
                        if (it % 11 == 0) x[3] = c.ut * V;
                        if (s) x[4] = q[4] * U(0.95, 1.05);
                    }
                    const fx::Gas G = fx::gas_of(g);
                    double f[8] = {0, 0, 0, 0, 0, 0, 0, 0};
                    bool ok;
                    if (mhd) {
                        fx::FluxI o;
                        ok = m == HLLD ? fx::mhd_face<true>(q, q + 7, G, o, f[7])
                                       : fx::mhd_face<false>(q, q + 7, G, o, f[7]);
                        const double t[7] = {o.m, o.mn, o.mt, o.e, o.bn, o.bt, o.bz};
                        for (int i = 0; i < 7; ++i) f[i] = t[i];
                    } else {
                        ok = m == HLLC ? fx::euler_face<false>(q, q + 7, G, f, f[7])
                                       : fx::euler_face<true>(q, q + 7, G, f, f[7]);
                        f[4] = f[5] = f[6] = 0;
                    }
                    if (!ok) { ++left; continue; }
                    ++taken;
                    L F[8];
                    flux((Solver)m, q, q + 7, g, F);
                    const L r = fmax(q[0], q[7]), S = F[7];
                    const L vt = fmax(fabs(q[3]), fabs(q[10])), W = fmaxl(S, vt);
                    const L bn = mhd ? fmax(fabs(q[4]), fabs(q[11])) : 0, B = 1;
                    const L sc[8] = {r * S, r * S * S, r * S * W, r * S * W * W, S * B, S * B + vt * bn,
                                     S * B, S};
                    for (int i = 0; i < 8; ++i) {
                        const double d = (double)(fabsl((L)f[i] - F[i]) / sc[i]);
                        if (!(d <= worst)) worst = d;
                    }
                }
                printf("%s %s %g taken %ld left %ld worst %.3e\n", solver[m], c.name, mach, taken, left,
                       worst);
            }
}
