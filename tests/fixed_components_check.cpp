// Host check that the integer face solvers keep small components: an out-of-plane field, a
// transverse velocity and field together, or a transverse velocity alone (fluid solvers, and no
// normal field), 2^-k times the normal ones; a weak normal field, alone or with the transverse one (the
// field of the plane beside a strong field out of it).  Usage: fixed_components_check <faces per class>.  One
// line per solver, class and k: the faces taken and left, and the largest error of the transverse
// momentum over density x fan speed x the transverse speed v (v plus b / sqrt(density) of the
// transverse field b where a normal field couples the two, times its 2^-k), of the transverse field over
// fan speed x b (or b + sqrt(density) v, as above), of the z field over fan speed x field and of the normal field over
// fan speed x normal field.
#define main ordinary_faces
#include "fixed_check.cpp"
#undef main

int main(int argc, char** argv) {
    const long n = argc > 1 ? atol(argv[1]) : 20000;
    std::mt19937_64 R(20260111);
    auto U = [&](double a, double b) { return a + (b - a) * (double)(R() >> 11) * 0x1p-53; };
    const char* solver[] = {"hllc", "hll", "hlld", "hllc_mhd"};
    // which components are small: transverse velocity, transverse field, z field, normal field
    struct { const char* name; bool v, t, z, n, nofield; double mach; } cls[] = {
        {"z_field", 0, 0, 1, 0, 0, 0.5},    {"z_field_fast", 0, 0, 1, 0, 0, 3},
        {"transverse", 1, 1, 0, 0, 0, 0.5}, {"transverse_fast", 1, 1, 0, 0, 0, 3},
        {"all", 1, 1, 1, 0, 0, 0.5},        {"velocity_across", 1, 0, 0, 0, 1, 0.5},
        {"normal", 0, 0, 0, 1, 0, 0.5},     {"in_plane", 0, 1, 0, 1, 0, 0.5},
        {"in_plane_fast", 0, 1, 0, 1, 0, 3}};
    for (int m = 0; m < 4; ++m)
        for (const auto& c : cls)
            for (int k : {0, 7, 14, 27, 40, 100}) {
                const bool mhd = m >= HLLD;
                if (!mhd && !c.v) continue;
                long taken = 0, left = 0;
                double worst = 0;
                for (long it = 0; it < n; ++it) {
                    const double g = it & 1 ? 1.4 : 5.0 / 3.0, w = std::ldexp(1.0, -k);
                    const double u = c.mach * U(-1, 1);
                    double q[14];
                    for (int s = 0; s < 2; ++s) {
                        double* x = q + 7 * s;
                        x[0] = U(0.8, 1.3);
                        x[1] = U(0.5, 0.8);
                        x[2] = u + 0.3 * U(-1, 1);
                        x[3] = (c.v ? w : 1) * U(-1, 1);
                        x[4] = c.nofield ? 0 : (c.n ? w : 1) * 0.7 * U(-1, 1);
                        x[5] = (c.t ? w : 1) * U(-1, 1);
                        x[6] = (c.z ? w : 1) * U(-1, 1);
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
                    const L vt = fmax(fabs(q[3]), fabs(q[10]));
                    const L bn = mhd ? fmax(fabs(q[4]), fabs(q[11])) : 0;
                    const L bt = mhd ? fmax(fabs(q[5]), fabs(q[12])) : 0;
                    const L bz = mhd ? fmax(fabs(q[6]), fabs(q[13])) : 0;
                    const L w1 = bn > 0 ? (c.n ? w : 1) : 0, root = sqrtl(r);
                    const L sc[8] = {r * S, r * S * S, r * S * (vt + w1 * bt / root), r * S * S * S,
                                     S * bn, S * (bt + w1 * root * vt), S * bz, S};
                    for (int i = 0; i < 8; ++i) {
                        const double d = (double)(fabsl((L)f[i] - F[i]) / (sc[i] + (L)0x1p-1000));
                        if (!(d <= worst)) worst = d;
                    }
                }
                printf("%s %s %d taken %ld left %ld worst %.3e\n", solver[m], c.name, k, taken, left,
                       worst);
            }
}
