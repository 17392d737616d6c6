// Host check of the integer MHD face solvers with components of independent sizes: transverse velocity,
// normal, transverse and z field from 1 down to 10^-range of the others.  Usage:
// fixed_exponents_check <faces>.  One line per solver and range: the faces taken and left, the
// largest error of a component over its natural scale (transverse momentum: density x fan speed x
// transverse speed + normal x transverse field; transverse field: fan speed x field + transverse speed x
// normal field; z and normal field: fan speed x field), and the share of faces above 1e-14 of it.
#define main ordinary_faces
#include "fixed_check.cpp"
#undef main

int main(int argc, char** argv) {
    const long n = argc > 1 ? atol(argv[1]) : 20000;
    for (int m = HLLD; m <= HLLC_MHD; ++m)
        for (double range : {3., 12., 40., 290.}) {
            std::mt19937_64 R(20260117);
            auto U = [&](double a, double b) { return a + (b - a) * (double)(R() >> 11) * 0x1p-53; };
            long taken = 0, left = 0, above = 0;
            double worst = 0;
            for (long it = 0; it < n; ++it) {
                const double g = it & 1 ? 1.4 : 5.0 / 3.0;
                const double u = U(-1, 1) * (it % 3 == 0 ? 3 : 0.5);
                double size[7], q[14];
                for (int k = 3; k < 7; ++k)
                    size[k] = U(0, 1) < 0.3 ? 1 : std::pow(10.0, U(-range, k == 3 ? 0 : 0.3));
                for (int s = 0; s < 2; ++s) {
                    double* x = q + 7 * s;
                    x[0] = U(0.8, 1.3);
                    x[1] = U(0.5, 0.8);
                    x[2] = u + U(-0.3, 0.3);
                    for (int k = 3; k < 7; ++k)
                        x[k] = size[k] * U(0.5, 1) * (it >> k & 1 ? -1 : 1) * (U(0, 1) < 0.1 ? -1 : 1);
                    if (U(0, 1) < 0.1) x[4] = 0;
                }
                const fx::Gas G = fx::gas_of(g);
                fx::FluxI o;
                double speed;
                if (!(m == HLLD ? fx::mhd_face<true>(q, q + 7, G, o, speed)
                                : fx::mhd_face<false>(q, q + 7, G, o, speed))) {
                    ++left;
                    continue;
                }
                ++taken;
                const double f[8] = {o.m, o.mn, o.mt, o.e, o.bn, o.bt, o.bz, speed};
                L F[8];
                flux((Solver)m, q, q + 7, g, F);
                auto big = [&](int k) { return fmaxl(fabsl((L)q[k]), fabsl((L)q[7 + k])); };
                const L r = big(0), S = F[7], vt = big(3), bn = big(4), bt = big(5), bz = big(6);
                const L sc[8] = {r * S, r * S * S, r * S * vt + bn * bt, r * S * S * S,
                                 S * bn, S * bt + vt * bn, S * bz, S};
                double e = 0;
                for (int k = 0; k < 8; ++k) {
                    const double d = (double)(fabsl((L)f[k] - F[k]) / (sc[k] + (L)0x1p-1010));
                    if (!(d <= e)) e = d;
                }
                if (!(e <= worst)) worst = e;
                above += !(e <= 1e-14);
            }
            printf("%s %g taken %ld left %ld worst %.3e above %.3e\n", m == HLLD ? "hlld" : "hllc_mhd",
                   range, taken, left, worst, (double)above / taken);
        }
}
