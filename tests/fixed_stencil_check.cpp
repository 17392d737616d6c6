// Host check of the states that a face takes from its four cells (face_states of gd_fixed.cuh) and
// of the flux between them, against long double.  Usage: fixed_stencil_check <faces per class>.
// The cells' values have 40 significant bits, so that c +- d/2 is exact in binary64 and the
// reference of fixed_check.cpp takes it as it is.  A class scales single cells or components of
// the stencil by powers of two.  One line per solver and class: the faces taken and left, the
// largest error of a face state over the larger of the two cells beside the face, and that of the
// flux over the scales of fixed_extremes_check with the velocities and fields of those two cells.
#define main ordinary_faces
#include "fixed_check.cpp"
#undef main
#include <cstring>

static double round40(double x) {
    int e;
    const double m = std::frexp(x, &e);
    return std::ldexp(std::nearbyint(std::ldexp(m, 40)), e - 40);
}
static double minmod(double a, double b) {
    return a * b <= 0 ? 0 : std::fabs(a) < std::fabs(b) ? a : b;
}

template <int NF, bool HLLD_OR_HLL>
static bool solve(const double (*c)[7], const fx::Gas& G, fx::i64* a, fx::i64* b, int* top,
                  double* f) {
    fx::i64 q[4 * NF];
    fx::Keys<NF> k[4];
    for (int i = 0; i < 4; ++i) fx::cell_units<NF>(c[i], q + i * NF, 1, k[i]);
    if (!fx::face_states<NF, 2>(q + 2 * NF, NF, 1, k + 2, 1, true, a, b, top)) return false;
    bool speed;
    if constexpr (NF == 4) {
        f[4] = f[5] = f[6] = 0;
        return fx::euler_flux<HLLD_OR_HLL>(a, b, top, G, f, f[7], speed, false);
    } else {
        fx::FluxI o;
        if (!fx::mhd_face_flux<HLLD_OR_HLL>(a, b, top, G, o, f[7], speed, false)) return false;
        const double t[7] = {o.m, o.mn, o.mt, o.e, o.bn, o.bt, o.bz};
        std::memcpy(f, t, sizeof t);
        return true;
    }
}

int main(int argc, char** argv) {
    const long n = argc > 1 ? atol(argv[1]) : 20000;
    std::mt19937_64 R(20260109);
    auto U = [&](double a, double b) { return a + (b - a) * (double)(R() >> 11) * 0x1p-53; };
    const char* solver[] = {"hllc", "hll", "hlld", "hllc_mhd"};
    // exponents by which the outer cells' vectors, their densities and pressures, the transverse
    // velocities of all cells and their fields are scaled
    struct { const char* name; int vec, gas, vt, b; } cls[] = {
        {"smooth", 0, 0, 0, 0},        {"strong_neighbour_4", 4, 0, 0, 0},
        {"strong_neighbour_12", 12, 0, 0, 0}, {"strong_neighbour_40", 40, 0, 0, 0},
        {"dense_neighbour", 0, 6, 0, 0}, {"thin_neighbour", 0, -30, 0, 0},
        {"weak_fields", 0, 0, 0, -40}, {"weak_neighbour", -40, 0, 0, 0},
        {"slow_across", 0, 0, -40, 0}, {"all_weak", 20, 0, -40, -40}};
    for (int m = 0; m < 4; ++m)
        for (const auto& c : cls) {
            const bool mhd = m >= HLLD;
            const int nf = mhd ? 7 : 4;
            long taken = 0, left = 0;
            double worst_state = 0, worst = 0;
            for (long it = 0; it < n; ++it) {
                const double g = it & 1 ? 1.4 : 5.0 / 3.0;
                double x[4][7];
                for (int i = 0; i < 4; ++i) {
                    const bool outer = i == 0 || i == 3;
                    for (int k = 0; k < 7; ++k) {
                        double v = k < 2 ? U(0.8, 1.6) : U(-0.6, 0.6);
                        if (outer && k >= 2) v = std::ldexp(v, c.vec);
                        if (outer && k < 2) v = std::ldexp(v, c.gas);
                        if (k == 3) v = std::ldexp(v, c.vt);
                        if (k >= 4) v = std::ldexp(v, c.b);
                        if ((it + k) % 17 == 0 && k >= 2) v = i % 2 ? 0.0 : -0.0;
                        x[i][k] = round40(v);
                    }
                }
                const fx::Gas G = fx::gas_of(g);
                fx::i64 a[7], b[7];
                int top[7];
                double f[8] = {0, 0, 0, 0, 0, 0, 0, 0};
                const bool ok = m == HLLC   ? solve<4, false>(x, G, a, b, top, f)
                                : m == HLL  ? solve<4, true>(x, G, a, b, top, f)
                                : m == HLLD ? solve<7, true>(x, G, a, b, top, f)
                                            : solve<7, false>(x, G, a, b, top, f);
                if (!ok) { ++left; continue; }
                ++taken;
                double q[14];
                for (int k = 0; k < nf; ++k) {
                    const double d = x[2][k] - x[1][k];
                    q[k] = x[1][k] + 0.5 * minmod(x[1][k] - x[0][k], d);
                    q[7 + k] = x[2][k] - 0.5 * minmod(d, x[3][k] - x[2][k]);
                    const L sc = fmaxl(fabsl(x[1][k]), fabsl(x[2][k])) + (L)0x1p-1000;
                    const L ea = fabsl(ldexpl((L)a[k], top[k] - 61) - q[k]) / sc;
                    const L eb = fabsl(ldexpl((L)b[k], top[k] - 61) - q[7 + k]) / sc;
                    worst_state = fmax(worst_state, (double)fmaxl(ea, eb));
                }
                L F[8];
                flux((Solver)m, q, q + 7, g, F);
                const L r = fmax(q[0], q[7]), S = F[7], E = r * S * S;
                const L vt = fmax(fabs(x[1][3]), fabs(x[2][3]));
                L B = 0;
                for (int i = 1; i < 3; ++i)
                    for (int k = 4; k < nf; ++k) B = fmaxl(B, fabsl(x[i][k]));
                const L sc[8] = {r * S, E, r * S * (mhd ? fmaxl(S, vt) : vt), E * S, B * S, B * S,
                                 B * S, S};
                for (int k = 0; k < 8; ++k) {
                    const double d = (double)(fabsl((L)f[k] - F[k]) / (sc[k] + (L)0x1p-1000));
                    if (!(d <= worst)) worst = d;
                }
            }
            printf("%s %s taken %ld left %ld state %.3e flux %.3e\n", solver[m], c.name, taken, left,
                   worst_state, worst);
        }
}
