// Host check of the integer face solvers at the ends of their range: densities and pressures at
// both ends of the accepted exponents, velocities and fields down to the smallest numbers, against
// the long double fluxes of fixed_check.cpp.  Usage: fixed_extremes_check <faces per class>.  One
// line per solver and class, as there; the error of a component is over the scale of fixed_check,
// of the fluid solvers' transverse momentum over density x fan speed x transverse speed.
#define main ordinary_faces
#include "fixed_check.cpp"
#undef main

int main(int argc, char** argv) {
    const long n = argc > 1 ? atol(argv[1]) : 20000;
    std::mt19937_64 R(20260107);
    auto U = [&](double a, double b) { return a + (b - a) * (double)(R() >> 11) * 0x1p-53; };
    const char* solver[] = {"hllc", "hll", "hlld", "hllc_mhd"};
    // density, pressure, velocity (0: of the order of the speed of sound), field over sqrt(p)
    struct { const char* name; double r, p, v, b; } cls[] = {
        {"interstellar", 1e-28, 1e-15, 1e-285, 1},     {"interstellar_weak", 1e-28, 1e-15, 1e-285, 1e-280},
        {"small", 1e-36, 1e-36, 1e-272, 1},            {"small_both", 1e-24, 1e-12, 1e-280, 1e-270},
        {"low_end", 0x1p-127, 0x1p-127, 0, 1},         {"high_end", 0x1p126, 0x1p126, 0, 1},
        {"cold", 0x1p126, 0x1p-127, 0, 1},             {"hot", 0x1p-127, 0x1p126, 0, 1},
        {"rest_low", 0x1p-127, 0x1p-127, 1e-90, 1e-70}, {"below_normal", 1, 1, 1e-310, 1e-309}};
    for (int m = 0; m < 4; ++m)
        for (const auto& c : cls) {
            const bool mhd = m >= HLLD;
            long taken = 0, left = 0;
            double worst = 0;
            for (long it = 0; it < n; ++it) {
                const double g = it & 1 ? 1.4 : 5.0 / 3.0;
                const double v = c.v > 0 ? c.v : 0.7 * std::sqrt(c.p / c.r);
                double q[14];
                for (int s = 0; s < 2; ++s) {
                    double* x = q + 7 * s;
                    x[0] = c.r * exp(U(-0.2, 0.2));
                    x[1] = c.p * exp(U(-0.2, 0.2));
                    x[2] = v * U(-1, 1);
                    x[3] = v * U(-1, 1);
                    for (int k = 4; k < 7; ++k) x[k] = c.b * std::sqrt(c.p) * U(-1, 1);
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
                const L r = fmax(q[0], q[7]), S = F[7], E = r * S * S;
                const L vt = fmax(fabs(q[3]), fabs(q[10]));
                const L B = S * c.b * std::sqrt(c.p);
                const L sc[8] = {r * S, E, r * S * (mhd ? fmaxl(S, vt) : vt), E * S, B, B, B, S};
                for (int k = 0; k < 8; ++k) {
                    const double d = (double)(fabsl((L)f[k] - F[k]) / (sc[k] + (L)0x1p-1074));
                    if (!(d <= worst)) worst = d;
                }
            }
            printf("%s %s taken %ld left %ld worst %.3e\n", solver[m], c.name, taken, left, worst);
        }
}
