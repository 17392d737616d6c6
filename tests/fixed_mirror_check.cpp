// Host check of the integer MHD face solvers at a mirror: the state above the face is that below it
// with the normal velocity and a part of the field reversed (the boundaries at x = 0 and on the axis),
// so that the contact stands exactly on the face, where a flux may jump between its two sides: the
// side below is the one taken (S_M >= 0).  Usage: fixed_mirror_check <faces per class>.  One line per
// solver and class: the faces taken and left, and the largest error of a component over density x fan
// speed^k or field x fan speed.
#define main ordinary_faces
#include "fixed_check.cpp"
#undef main

int main(int argc, char** argv) {
    const long n = argc > 1 ? atol(argv[1]) : 20000;
    std::mt19937_64 R(20260119);
    auto U = [&](double a, double b) { return a + (b - a) * (double)(R() >> 11) * 0x1p-53; };
    const char* solver[] = {"hllc", "hll", "hlld", "hllc_mhd"};
    struct { const char* name; double n, t, z, p; } cls[] = {
        {"mirror", -1, -1, 1, 0.7}, {"axis", 1, 1, -1, 0.7}, {"wall", -1, 1, 1, 0.7},
        {"cold_mirror", -1, -1, 1, 1e-9}, {"tenuous_axis", 1, 1, -1, 1e-6}};
    for (int m = HLLD; m <= HLLC_MHD; ++m)
        for (const auto& c : cls) {
            long taken = 0, left = 0;
            double worst = 0;
            for (long it = 0; it < n; ++it) {
                const double g = it & 1 ? 1.4 : 5.0 / 3.0, v = std::sqrt(c.p);
                double q[14];
                q[0] = U(0.5, 2);
                q[1] = c.p * U(0.5, 2);
                q[2] = v * U(-1, 1);
                q[3] = v * U(-1, 1);
                for (int k = 4; k < 7; ++k) q[k] = v * U(-1, 1);
                if (it % 5 == 0) q[4 + it / 5 % 3] = 0;
                const double s[7] = {1, 1, -1, 1, c.n, c.t, c.z};
                for (int k = 0; k < 7; ++k) q[7 + k] = s[k] * q[k];
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
                const L r = q[0], S = F[7], B = v;
                const L sc[8] = {r * S, r * S * S, r * S * S, r * S * S * S, S * B, S * B, S * B, S};
                for (int k = 0; k < 8; ++k) {
                    const double d = (double)(fabsl((L)f[k] - F[k]) / sc[k]);
                    if (!(d <= worst)) worst = d;
                }
            }
            printf("%s %s taken %ld left %ld worst %.3e\n", solver[m], c.name, taken, left, worst);
        }
}
