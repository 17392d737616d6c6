// gd_fast_mhd.cu -- fused minmod-TVD + HLLD / HLLC-MHD + Powell-source update for 2-D ideal
// MHD, face-once tiles (same phase structure as gd_fast_euler.cu: load, slopes, faces,
// update), and its forward-mode tangent.
//
// The step's slopes and faces run in scaled 64-bit integers (gd_fixed_mhd.cuh), as in
// gd_fast_euler.cu: 92 FP64 operations per cell against 448.  A face whose states or fan leave the
// integers' range is solved in FP64 from the cells themselves.  The tangent's tile is floating
// point throughout; it and the flux are templates on the scalar type, and `Dual` (gd_dual.cuh)
// gives the tangent (JVP), with the dt held fixed and derivatives taken along the branches the
// values take.
//
// Field units.  The reference stores Gaussian B and divides by sqrt(4 pi) inside every flux
// call (Gas_Dinamic.cu:970-976), multiplying the field fluxes back (:1497-1499).  Here the
// field is converted once per cell when the tile is loaded, b = B / sqrt(4 pi), the whole
// step runs in these units, and B = b * sqrt(4 pi) is stored.  In these units the Powell
// terms of the reference update (kernel.cu:2641-2648), (B/4pi) Pdiv_B, (v.B/4pi) Pdiv_B and
// v Pdiv_B, become b Pdiv_b, (v.b) Pdiv_b and v Pdiv_b, and |B|^2/8pi becomes |b|^2/2.
//
// Reference semantics kept: primitive reconstruction of all seven fields with the rho/p
// fallback (kernel.cu:2407-2548); wave speeds SL = min(u) - max(cf), SR = max(u) + max(cf),
// SM and p_T* (Gas_Dinamic.cu:1062-1075); HLL-averaged field; HLLD star and double-star
// states with the |tt| >= 1e-5 and |bn| > 1e-6 guards (:1306-1430) and the six-region
// selection (:1434-1484), or the HLLC-MHD states (:1137-1302); normal-field flux
// -max(|SL|,|SR|) (bn_R - bn_L) (:1488-1490); Powell divergence from cell-centred B
// (kernel.cu:2568-2604); axisymmetric sources (kernel.cu:2615-2648); floors rho <= 0 ->
// old rho, p <= 0 -> 1e-6; dt = min over faces of krit*rad/max(|SL|,|SR|), rad = dx on
// x-faces (kernel.cu:2560).
#include <type_traits>

#include "gd_dual.cuh"
#include "gd_fixed_mhd.cuh"
#include "gd_internal.cuh"
#include "gd_kernels.h"
#include "gd_mhd_flux.cuh"

namespace gd {
namespace {

constexpr int TX = 32;
constexpr int kNT = 384;  // threads of the step (see kTY)
// Threads where every tile has an SM to itself (Params::few_tiles): the step is one tile's latency, and
// 768 threads take its 747 faces in one round: 31.5 against 37.1 us at 64x48, 30.5 against 37.1 at
// 320x165 (150 tiles).  At 160 tiles 53.8 against 51.5: there the 384-thread tiles stay.
constexpr int kNTFew = 768;
// The tangent's: one CTA per SM.  20 tangent steps at 512^2 take 16.1 ms with 256 threads, 15.0
// with 384, 15.3 with 576.
constexpr int NTDual = 384;
constexpr int NF = 7;  // rho, p, vx, vy, bx, by, bz

// ---- state access: planes of doubles for the step, value + tangent planes for the JVP ----

struct DualCPlanes {
    CPlanes v, d;
};
struct DualPlanes {  // the tangent alone: the values are the recorded run's
    Planes d;
};

__device__ __forceinline__ void load_state(const Params& P, const CPlanes& in, int gx, int gy,
                                           double* v) {
    fetch_cell<NF>(P, in, gx, gy, v);
}

// Tangent of a ghost value: the linear part of the boundary condition.  Copies and sign
// flips carry the derivative; constants (ambient) and the active outflow clamp have none.
__device__ __forceinline__ void load_state(const Params& P, const DualCPlanes& in, int gx,
                                           int gy, Dual* v) {
    double a[NF], b[NF];
    fetch_cell<NF>(P, in.v, gx, gy, a);
    fetch_cell<NF>(P, in.d, gx, gy, b);
    int bc = -1;
    if (gx < 0 || gx >= P.N) bc = gx < 0 ? P.bc[0] : P.bc[1];
    else if (gy < 0 || gy >= P.M) bc = gy < 0 ? P.bc[2] : P.bc[3];
    if (bc == GD_BC_AMBIENT || bc == GD_BC_AMBIENT_KEEPB) {
        for (int f = 0; f < (bc == GD_BC_AMBIENT ? NF : 4); ++f) b[f] = 0.0;
    } else if (bc == GD_BC_OUTFLOW) {
        double raw[NF];
        CPlanes plain = in.v;
        int sx = gx < 0 ? 0 : (gx >= P.N ? P.N - 1 : gx);
        int sy = gy < 0 ? 0 : (gy >= P.M ? P.M - 1 : gy);
        raw[2] = plain.f[2][(long long)sy * P.N + sx];
        if (raw[2] < 0) b[2] = 0.0;
    }
#pragma unroll
    for (int f = 0; f < NF; ++f) v[f] = Dual{a[f], b[f]};
}

__device__ __forceinline__ void store_state(const Planes& out, long long k, int f, double x) {
    store_f(out, f, k, x);
}
__device__ __forceinline__ void store_state2(const Planes& out, long long k, int f0, double a,
                                             double b) {
    store_pair(out, f0, k, a, b);
}
__device__ __forceinline__ void store_state(const DualPlanes& out, long long k, int f, Dual x);
__device__ __forceinline__ void store_state2(const DualPlanes& out, long long k, int f0, Dual a,
                                             Dual b) {
    store_state(out, k, f0, a);
    store_state(out, k, f0 + 1, b);
}
__device__ __forceinline__ void store_state(const DualPlanes& out, long long k, int f, Dual x) {
    out.d.f[f][k] = x.d;
}
__device__ __forceinline__ void copy_cell(const CPlanes& in, const Planes& out, long long k) {
#pragma unroll
    for (int f = 0; f < NF; ++f) store_f(out, f, k, load_f(in, f, k));
}
__device__ __forceinline__ void copy_cell(const DualCPlanes& in, const DualPlanes& out,
                                          long long k) {
#pragma unroll
    for (int f = 0; f < NF; ++f) out.d.f[f][k] = in.d.f[f][k];
}

// The tangent's tile.
template <class T, int ORDER, int TY>
struct SmemM {
    static constexpr int H = ORDER == 2 ? 2 : 1;
    static constexpr int SX = TX + 2 * H;
    static constexpr int SY = TY + 2 * H;
    static constexpr int kPrim = NF * SY * SX;
    static constexpr int kSlx = ORDER == 2 ? NF * TY * (TX + 2) : 0;
    static constexpr int kSly = ORDER == 2 ? NF * (TY + 2) * TX : 0;
    static constexpr int kFx = NF * TY * (TX + 1);
    static constexpr int kFy = NF * (TY + 1) * TX;
    static constexpr size_t bytes = sizeof(T) * (kPrim + kSlx + kSly + kFx + kFy);
};
// The step's tile: the cells' significands and keys (gd_fixed.cuh), and b_x and b_y of the tile's
// cells and of those beside them in x and in y.  The update reads the other values again from global
// memory: with all seven here (102 KB a tile) the rest of the L1 was too small for the face code's
// spills (vortex of 1024^2, four steps: 1.90 against 1.88 ms).
template <int ORDER, int TY>
struct ShapeInt {
    static constexpr int H = ORDER == 2 ? 2 : 1;
    static constexpr int SX = TX + 2 * H;
    static constexpr int SY = TY + 2 * H;
    static constexpr int kKey = 2 * SY * SX;
    static constexpr int kPrim = NF * SY * SX;
    static constexpr int kCell = 2 * TX * TY;
    static constexpr int kEdge = 2 * (TX + TY);
    static constexpr int kFx = NF * TY * (TX + 1);
    static constexpr int kFy = NF * (TY + 1) * TX;
    static constexpr size_t bytes = sizeof(double) * (kKey + kPrim + kCell + kEdge + kFx + kFy);
};

struct MhdTileResult {
    double umax_x, umax_y;
    bool any_active;
    unsigned int nfl_r, nfl_p, nbad;
};

// One face of a tile: faces 0 .. NFX-1 have an x normal, the rest a y normal.
template <int TY>
struct FaceM {
    static constexpr int NFX = (TX + 1) * TY, NFY = TX * (TY + 1), kAll = NFX + NFY;
    bool isx, used;
    int lx, ly;
    // used: inside the grid, and next to a cell that the step updates
    __device__ FaceM(const Params& P, int tx0, int ty0, int i) {
        isx = i < NFX;
        if (isx) {
            ly = i / (TX + 1);
            lx = i - ly * (TX + 1);
            used = tx0 + lx <= P.N && ty0 + ly < P.M;
        } else {
            const int j = i - NFX;
            ly = j / TX;
            lx = j - ly * TX;
            used = tx0 + lx < P.N && ty0 + ly <= P.M;
        }
        if (used && P.frozen)
            used = cell_active(P, tx0 + (isx ? lx - 1 : lx), ty0 + (isx ? ly : ly - 1)) ||
                   cell_active(P, tx0 + lx, ty0 + ly);
    }
    // field of the local frame's component f: x-face (n, t) = (x, y); y-face (n, t) = (y, x)
    __device__ __forceinline__ int field(int f) const {
        return isx || f < 2 || f == 6 ? f : (f < 4 ? 5 - f : 9 - f);
    }
    template <class T>
    __device__ __forceinline__ void store(T* fx, T* fy, const FluxM<T>& F) const {
        constexpr int sx = TY * (TX + 1), sy = (TY + 1) * TX;
        T* fo = isx ? fx + ly * (TX + 1) + lx : fy + ly * TX + lx;
        const int st = isx ? sx : sy;
        fo[0 * st] = F.m;
        fo[1 * st] = F.e;
        fo[2 * st] = isx ? F.mn : F.mt;
        fo[3 * st] = isx ? F.mt : F.mn;
        fo[4 * st] = isx ? F.bn : F.bt;
        fo[5 * st] = isx ? F.bt : F.bn;
        fo[6 * st] = F.bz;
    }
};

struct SpeedsM {
    double x, y;
    __device__ __forceinline__ void take(bool isx, double UU) {
        if (isx) x = max_nonneg(x, UU);
        else y = max_nonneg(y, UU);
    }
};

// the flux in floating point between two states of the local frame
template <class T>
__device__ __forceinline__ FluxM<T> float_flux(const Params& P, const T* qa, const T* qb, T& UU) {
    Side<T> A, B;
    side(A, qa[0], qa[1], qa[2], qa[3], qa[4], qa[5], qa[6], P);
    side(B, qb[0], qb[1], qb[2], qb[3], qb[4], qb[5], qb[6], P);
    return hlld_local(A, B, P.method, P, UU);
}
// the states on either side of a face, c + d/2 and c - d/2; rho and p fall back to the cell's
template <class T>
__device__ __forceinline__ void side_states(int f, T ca, T da, T cb, T db, T& a, T& b) {
    a = fma(0.5, da, ca);
    b = fma(-0.5, db, cb);
    if (f < 2) {
        a = le_zero(a) ? ca : a;
        b = le_zero(b) ? cb : b;
    }
}

// ---- U: update (kernel.cu:2606-2660 in Heaviside-Lorentz field units) --------------------------
// Written so that no product stands alone beside a sum: there is nothing for the compiler to contract
// in one kernel and not in another, and the step's kernels round alike.
// cell: a cell's values; jump: b_x across a cell in x and b_y
// in y, from its neighbours.  `aux` (T = double only; may be null) receives, per cell, the flux
// differences d[0..6] and the Powell term divb that the update used (planes of N*M), for the adjoint.
template <class T, int BT, int TY, class IN, class OUT, class CELL, class JUMP>
__device__ __forceinline__ void update_cells(const Params& P, const IN& in, const OUT& out, int tx0,
                                             int ty0, double T_do, int dt_only, const CELL& cell,
                                             const JUMP& jump, const T* fx, const T* fy,
                                             MhdTileResult& res, double* aux) {
    const int N = P.N, M = P.M;
    const double kx = imul<true>(T_do, P.inv_dx), ky = imul<true>(T_do, P.inv_dy);
    const double hkx = half_exact(kx), hky = half_exact(ky);  // 0.5 kx, 0.5 ky
    const bool axi = P.geometry == GD_AXISYM;
    bool any_active = false;
    unsigned int nfl_r = 0, nfl_p = 0, nbad = 0;
    for (int i = threadIdx.x; i < TX * TY; i += BT) {
        const int ly = i / TX, lx = i - ly * TX;
        const int gx = tx0 + lx, gy = ty0 + ly;
        if (gx >= N || gy >= M) continue;
        const long long k = (long long)gy * N + gx;
        if (P.frozen && !cell_active(P, gx, gy)) {  // the faces' own test
            if (!dt_only) copy_cell(in, out, k);
            continue;
        }
        any_active = true;
        if (dt_only) continue;
        T c[NF];
        cell(lx, ly, gx, gy, c);
        const T r = c[0], p = c[1], u = c[2], v = c[3], bx = c[4], by = c[5], bz = c[6];
        const T* fxc = fx + ly * (TX + 1) + lx;
        const T* fyc = fy + ly * TX + lx;
        T d[NF];
#pragma unroll
        for (int f = 0; f < NF; ++f) {
            const T* a = fxc + f * TY * (TX + 1);
            const T* b = fyc + f * (TY + 1) * TX;
            d[f] = fma(kx, a[1] - a[0], ky * (b[TX] - b[0]));
        }
        // Powell divergence from cell-centred field: dx dy div b (kernel.cu:2568-2604)
        T divb = fma(hkx, jump.x(lx, ly), mulx<true>(hky, jump.y(lx, ly)));  // T_do * div b
        const double iy = axi ? rcp_fast(fma((double)gy, P.dy, P.y0)) : 0.0;
        if (axi) divb = fma(T_do * by, iy, divb);                 // kernel.cu:2615
        if constexpr (std::is_same<T, double>::value) {
            if (aux != nullptr) {
                const long long KK = (long long)N * M;
#pragma unroll
                for (int f = 0; f < NF; ++f) aux[f * KK + k] = d[f];
                aux[7 * KK + k] = divb;
            }
        }
        const T ub = fma(u, bx, v * by);
        const T bb = fma(bz, bz, fma(by, by, bx * bx));
        const T K1 = fma(r, fma(u, u, v * v), bb);  // twice the kinetic and field energy
        T r2 = r - d[0];
        T mx2 = fma(r, u, -fma(bx, divb, d[2]));
        T my2 = fma(r, v, -fma(by, divb, d[3]));
        T bx2 = bx - fma(u, divb, d[4]);
        const T by2 = by - fma(v, divb, d[5]);
        const T bz2 = bz - d[6];
        T dE = fma(ub, divb, d[1]);
        if (axi) {
            // geometric sources / y (kernel.cu:2619-2648) in field units b
            const double ty = T_do * iy;
            r2 = fma(-ty * r, v, r2);
            mx2 = fma(-ty, fma(r * u, v, -bx * by), mx2);
            my2 = fma(-ty, fma(r * v, v, fma(bz, bz, -by * by)), my2);
            bx2 = fma(-ty, fma(v, bx, -by * u), bx2);
            dE = fma(ty, fma(fma(p, P.g_gm1, 0.5 * (K1 + bb)), v, -by * ub), dE);
        }
        if (le_zero(r2)) { r2 = r; ++nfl_r; }
        const T inv = rcp_fast(r2);
        const T u2 = mx2 * inv, v2 = my2 * inv;
        // p' = p - (gamma - 1) (d_E - (K - K') / 2): no sum of the whole energy to round
        const T K2 = fma(r2, fma(u2, u2, v2 * v2), fma(bz2, bz2, fma(by2, by2, bx2 * bx2)));
        T p2 = fma(P.hgm1, K1 - K2, fma(-P.gm1, dE, p));
        if (le_zero(p2)) { p2 = cst<T>(0.000001); ++nfl_p; }
        if (!finite_bits(r2) || !finite_bits(p2) || !finite_bits(u2) || !finite_bits(v2) ||
            !finite_bits(bx2) || !finite_bits(by2) || !finite_bits(bz2))
            ++nbad;
        store_state2(out, k, 0, r2, p2);
        store_state2(out, k, 2, u2, v2);
        store_state(out, k, 4, bx2 * kSpi4);
        store_state(out, k, 5, by2 * kSpi4);
        store_state(out, k, 6, bz2 * kSpi4);
    }
    res.any_active = any_active;
    res.nfl_r = nfl_r;
    res.nfl_p = nfl_p;
    res.nbad = nbad;
}

template <class T, int SX, int FS>
struct JumpFloat {
    const T* own;  // the tile's first cell
    __device__ __forceinline__ T x(int lx, int ly) const {
        const T* c = own + 4 * FS + ly * SX + lx;
        return c[1] - c[-1];
    }
    __device__ __forceinline__ T y(int lx, int ly) const {
        const T* c = own + 5 * FS + ly * SX + lx;
        return c[SX] - c[-SX];
    }
};

// The tangent's TX x TY tile at (tx0, ty0): load, slopes, faces, update, with IN/OUT
// DualCPlanes/DualPlanes for T = Dual.
// flux component slots in smem: 0 mass, 1 energy, 2 mom x, 3 mom y, 4 bx, 5 by, 6 bz
template <class T, int BT, int ORDER, int TY, class IN, class OUT>
__device__ __noinline__ void mhd_tile(const Params& P, const IN& in, const OUT& out, int tx0,
                                         int ty0, double T_do, int dt_only, T* smem,
                                         MhdTileResult& res, double* aux) {
    using S = SmemM<T, ORDER, TY>;
    constexpr int H = S::H, SX = S::SX, SY = S::SY;
    T* prim = smem;
    T* slx = prim + S::kPrim;
    T* sly = slx + S::kSlx;
    T* fx = sly + S::kSly;
    T* fy = fx + S::kFx;

    const int tid = threadIdx.x;
    const int N = P.N, M = P.M;

    // ---- L: tile + cross halo, field to Heaviside-Lorentz units --------------------------
    for (int i = tid; i < SY * SX; i += BT) {
        const int ly = i / SX, lx = i - ly * SX;
        const bool xh = lx < H || lx >= TX + H, yh = ly < H || ly >= TY + H;
        if (xh && yh) continue;
        const int gx = tx0 + lx - H, gy = ty0 + ly - H;
        T v[NF];
        if (gx >= -2 && gx < N + 2 && gy >= -2 && gy < M + 2 &&
            !((gx < 0 || gx >= N) && (gy < 0 || gy >= M))) {
            load_state(P, in, gx, gy, v);
        } else {
#pragma unroll
            for (int f = 0; f < NF; ++f) v[f] = cst<T>(f < 2 ? 1.0 : 0.0);  // never used
        }
        v[4] = v[4] * kInvSpi4;
        v[5] = v[5] * kInvSpi4;
        v[6] = v[6] * kInvSpi4;
#pragma unroll
        for (int f = 0; f < NF; ++f) prim[(f * SY + ly) * SX + lx] = v[f];
    }
    __syncthreads();

    // ---- S: slopes ---------------------------------------------------------------------------
    // a thread takes a run of G cells, so neighbouring slopes share their difference
    if constexpr (ORDER == 2) {
        constexpr int GX = (TX + 2) % 3 == 0 ? 3 : 2, GY = (TY + 2) % 3 == 0 ? 3 : 2;
        constexpr int NGX = (TX + 2) / GX, NGY = (TY + 2) / GY;
        static_assert((TX + 2) % GX == 0 && (TY + 2) % GY == 0, "slope runs tile the rows");
        for (int i = tid; i < TY * NGX; i += BT) {
            const int ly = i / NGX, c0 = (i - ly * NGX) * GX;
            const T* row = prim + (ly + H) * SX + (c0 - 1 + H);
#pragma unroll
            for (int f = 0; f < NF; ++f) {
                const T* q = row + f * SY * SX;
                T* o = slx + (f * TY + ly) * (TX + 2) + c0;
                T dl = q[0] - q[-1];
#pragma unroll
                for (int j = 0; j < GX; ++j) {
                    const T dr = q[j + 1] - q[j];
                    o[j] = minmod(dl, dr);
                    dl = dr;
                }
            }
        }
        for (int i = tid; i < NGY * TX; i += BT) {
            const int g = i / TX, lx = i - g * TX, r0 = g * GY;
            const T* col = prim + (r0 - 1 + H) * SX + (lx + H);
#pragma unroll
            for (int f = 0; f < NF; ++f) {
                const T* q = col + f * SY * SX;
                T* o = sly + (f * (TY + 2) + r0) * TX + lx;
                T dl = q[0] - q[-SX];
#pragma unroll
                for (int j = 0; j < GY; ++j) {
                    const T dr = q[(j + 1) * SX] - q[j * SX];
                    o[j * TX] = minmod(dl, dr);
                    dl = dr;
                }
            }
        }
        __syncthreads();
    }

    // ---- F: faces ----------------------------------------------------------------------------
    SpeedsM u{0.0, 0.0};
    for (int i = tid; i < FaceM<TY>::NFX + FaceM<TY>::NFY; i += BT) {
        const FaceM<TY> w(P, tx0, ty0, i);
        if (!w.used) continue;
        const int lx = w.lx, ly = w.ly;
        const T* pb = prim + (ly + H) * SX + (lx + H);
        const T* pa = pb - (w.isx ? 1 : SX);
        T qa[NF], qb[NF], UU;
#pragma unroll
        for (int f = 0; f < NF; ++f) {
            const int g = w.field(f);
            qa[f] = pa[g * SY * SX];
            qb[f] = pb[g * SY * SX];
            if (ORDER == 2) {
                T da, db;
                if (w.isx) {
                    da = slx[(g * TY + ly) * (TX + 2) + lx];
                    db = slx[(g * TY + ly) * (TX + 2) + lx + 1];
                } else {
                    da = sly[(g * (TY + 2) + ly) * TX + lx];
                    db = sly[(g * (TY + 2) + ly + 1) * TX + lx];
                }
                side_states(f, qa[f], da, qb[f], db, qa[f], qb[f]);
            }
        }
        w.store(fx, fy, float_flux(P, qa, qb, UU));
        u.take(w.isx, value_of(UU));
    }
    __syncthreads();

    const T* own = prim + H * SX + H;
    const auto cell = [&](int lx, int ly, int, int, T* v) {
#pragma unroll
        for (int f = 0; f < NF; ++f) v[f] = own[f * SY * SX + ly * SX + lx];
    };
    update_cells<T, BT, TY>(P, in, out, tx0, ty0, T_do, dt_only, cell,
                            JumpFloat<T, SX, SY * SX>{own}, fx, fy, res, aux);
    res.umax_x = u.x;
    res.umax_y = u.y;
}

// ---- The step's tile: face work in 64-bit integers --------------------------------------------
//
// HLLD takes about 150 binary64 operations a face; on the FP64 pipe, at 64 cycles of a sub-
// partition each, they held the tile to 35 000 cycles per 32 cells.  Here the cells of the tile
// and its halo are significands and exponents (gd_fixed.cuh), a face shifts its stencil to units of
// its own, slopes and face states are adds and selects, and the flux is fx::mhd_flux.  The FP64 pipe
// keeps the conversion of the fluxes and the update.  Bound by the latency of the integer chains (ALU
// 50 %, issue 47 %, FP64 37 %).
template <int ORDER, int TY>
struct MemInt {
    using S = ShapeInt<ORDER, TY>;
    using Key = fx::Keys<NF>;
    static_assert(sizeof(Key) == 2 * sizeof(double), "keys take two doubles a cell");
    Key* key;      // [SY][SX]
    fx::i64* q;    // [NF][SY][SX]
    double* cell;  // [2][TY][TX]  b_x, b_y
    double* edgex;  // [2][TY]  b_x of the cells at x = -1 and TX
    double* edgey;  // [2][TX]  b_y of the cells at y = -1 and TY
    double *fx, *fy;
    __device__ explicit MemInt(double* smem)
        : key(reinterpret_cast<Key*>(smem)), q(reinterpret_cast<fx::i64*>(smem + S::kKey)),
          cell(smem + S::kKey + S::kPrim), edgex(cell + S::kCell), edgey(edgex + 2 * TY),
          fx(edgey + 2 * TX), fy(fx + S::kFx) {}
};

// One compiled body for every kernel, so that a face left to floating point has the same bits
// whichever kernel solves it.
__device__ __noinline__ FluxM<double> float_flux_of(const Params& P, const double* qa,
                                                    const double* qb, double& UU) {
    return float_flux(P, qa, qb, UU);
}
__device__ __forceinline__ void load_cell(const Params& P, const CPlanes& in, int gx, int gy,
                                          double* v) {
    load_state(P, in, gx, gy, v);
#pragma unroll
    for (int f = 4; f < NF; ++f) v[f] = __dmul_rn(v[f], kInvSpi4);
}

// The faces that the integer solver left, in floating point from the cells themselves.  Out of
// line and after the loop over the faces, so that it takes no registers from it; a list for the
// whole block, so that a few faces of each warp cost what they are (an HLLD step of 1024^2 cells with
// densities and pressures at random over 2^6: 776 us, 1549 with each thread redoing its own).
template <int ORDER, int TY, int NT>
__device__ __noinline__ void faces_left(const Params& P, const CPlanes& in, double* smem, int tx0,
                                        int ty0, const LeftFaces<FaceM<TY>::kAll>& left,
                                        SpeedsM& u) {
    const MemInt<ORDER, TY> t(smem);
    for (unsigned int k = threadIdx.x; k < left.n; k += NT) {
        const FaceM<TY> w(P, tx0, ty0, left.face(k));
        const int gx = tx0 + w.lx, gy = ty0 + w.ly, sx = w.isx ? 1 : 0, sy = w.isx ? 0 : 1;
        double c[4][NF], qa[NF], qb[NF], UU;
        load_cell(P, in, gx - sx, gy - sy, c[1]);
        load_cell(P, in, gx, gy, c[2]);
        if (ORDER == 2) {
            load_cell(P, in, gx - 2 * sx, gy - 2 * sy, c[0]);
            load_cell(P, in, gx + sx, gy + sy, c[3]);
        }
#pragma unroll
        for (int f = 0; f < NF; ++f) {
            double a = c[1][f], b = c[2][f];
            if (ORDER == 2) {
                const double d = b - a;
                side_states(f, a, minmod(a - c[0][f], d), b, minmod(d, c[3][f] - b), a, b);
            }
            qa[w.field(f)] = a;  // the swap is its own inverse
            qb[w.field(f)] = b;
        }
        w.store(t.fx, t.fy, float_flux_of(P, qa, qb, UU));
        if (left.no_speed(k)) u.take(w.isx, UU);
    }
}

template <int TY>
struct JumpCells {
    const double *cell, *edgex, *edgey;
    __device__ __forceinline__ double x(int lx, int ly) const {
        const double* c = cell + ly * TX + lx;
        return (lx < TX - 1 ? c[1] : edgex[TY + ly]) - (lx > 0 ? c[-1] : edgex[ly]);
    }
    __device__ __forceinline__ double y(int lx, int ly) const {
        const double* c = cell + TX * TY + ly * TX + lx;
        return (ly < TY - 1 ? c[TX] : edgey[TX + lx]) - (ly > 0 ? c[-TX] : edgey[lx]);
    }
};

// One tile of the step.  Every thread of the block must call it.
template <bool HLLD, int ORDER, int TY, int NT>
__device__ __forceinline__ void step_tile(const Params& P, const CPlanes& in, const Planes& out,
                                          int tx0, int ty0, double T_do, int dt_only,
                                          double* smem, MhdTileResult& res, double* aux) {
    using S = ShapeInt<ORDER, TY>;
    using fx::i64;
    constexpr int H = S::H, SX = S::SX, SY = S::SY, FS = SY * SX;
    const MemInt<ORDER, TY> t(smem);
    __shared__ LeftFaces<FaceM<TY>::kAll> left;
    const int tid = threadIdx.x, N = P.N, M = P.M;
    if (tid == 0) left.n = 0;
    for (int i = tid; i < FS; i += NT) {
        const int ly = i / SX - H, lx = i % SX - H;
        const bool xh = lx < 0 || lx >= TX, yh = ly < 0 || ly >= TY;
        const int gx = tx0 + lx, gy = ty0 + ly;
        if ((xh && yh) || gx < -2 || gx >= N + 2 || gy < -2 || gy >= M + 2 ||
            ((gx < 0 || gx >= N) && (gy < 0 || gy >= M)))
            continue;  // no face reads it
        double v[NF];
        load_cell(P, in, gx, gy, v);
        fx::cell_units<NF>(v, t.q + i, FS, t.key[i]);
        if (!xh && !yh) {
#pragma unroll
            for (int f = 0; f < 2; ++f) t.cell[(f * TY + ly) * TX + lx] = v[4 + f];
        } else if (lx == -1 || lx == TX) {
            t.edgex[(lx == TX ? TY : 0) + ly] = v[4];
        } else if (ly == -1 || ly == TY) {
            t.edgey[(ly == TY ? TX : 0) + lx] = v[5];
        }
    }
    __syncthreads();

    SpeedsM u{0.0, 0.0};
    for (int i = tid; i < FaceM<TY>::kAll; i += NT) {
        const FaceM<TY> w(P, tx0, ty0, i);
        if (!w.used) continue;
        const int c = (w.ly + H) * SX + w.lx + H, st = w.isx ? 1 : SX;
        i64 a[NF], b[NF];
        int top[NF];
        double UU;
        fx::FluxI F;
        bool speed_ok = false, done = false;
        if (P.gas.room >= 0 &&
            fx::face_states<NF, ORDER>(t.q + c, st, FS, t.key + c, st, w.isx, a, b, top))
            done = fx::mhd_face_flux<HLLD>(a, b, top, P.gas, F, UU, speed_ok, dt_only);
        if (speed_ok) u.take(w.isx, UU);
        if (!done) left.add(i, speed_ok);
        else if (!dt_only)
            w.store(t.fx, t.fy, FluxM<double>{F.m, F.mn, F.mt, F.e, F.bn, F.bt, F.bz});
    }
    __syncthreads();
    if (left.n != 0) {
        faces_left<ORDER, TY, NT>(P, in, smem, tx0, ty0, left, u);
        __syncthreads();
    }

    const auto cell = [&](int, int, int gx, int gy, double* v) { load_cell(P, in, gx, gy, v); };
    update_cells<double, NT, TY>(P, in, out, tx0, ty0, T_do, dt_only, cell,
                                 JumpCells<TY>{t.cell, t.edgex, t.edgey}, t.fx, t.fy, res, aux);
    res.umax_x = u.x;
    res.umax_y = u.y;
}

template <int ORDER, int TY, bool HLLD, int NT>
__global__ void __launch_bounds__(NT, NT == kNT ? 2 : 1) mhd_fast_kernel(const __grid_constant__ Params P,
                                                      const __grid_constant__ CPlanes in,
                                                      const __grid_constant__ Planes out,
                                                      const double* __restrict__ T_do_ptr,
                                                      unsigned long long* T_bits, Scalars* rot,
                                                      Scalars* ctr, int dt_only, double* aux) {
    extern __shared__ __align__(16) double smem[];
    MhdTileResult r;
    step_tile<HLLD, ORDER, TY, NT>(P, in, out, blockIdx.x * TX, (blockIdx.y + P.tile_row0) * TY,
                                   *T_do_ptr, dt_only, smem, r, aux);
    if (ctr != nullptr && (r.nfl_r | r.nfl_p | r.nbad)) {
        if (r.nfl_r) atomicAdd(&ctr->rho_floor, (unsigned long long)r.nfl_r);
        if (r.nfl_p) atomicAdd(&ctr->p_floor, (unsigned long long)r.nfl_p);
        if (r.nbad) atomicAdd(&ctr->nonfinite, (unsigned long long)r.nbad);
    }
    block_dt_and_rotate<NT>(P, r.umax_x, r.umax_y, r.any_active, T_bits, rot, P.tile_nblocks);
}

// Tangent of one step: (U, dU) -> dU' with the dt read from *T_do_ptr (held fixed).
template <int ORDER, int TY>
__global__ void __launch_bounds__(NTDual) mhd_tangent_kernel(const __grid_constant__ Params P,
                                                         CPlanes in, CPlanes din,
                                                         Planes dout,
                                                         const double* __restrict__ T_do_ptr) {
    extern __shared__ __align__(16) double smem[];
    MhdTileResult r;
    const DualCPlanes I{in, din};
    const DualPlanes O{dout};
    mhd_tile<Dual, NTDual, ORDER, TY>(P, I, O, blockIdx.x * TX, blockIdx.y * TY, *T_do_ptr, 0,
                              reinterpret_cast<Dual*>(smem), r, nullptr);
}

// 32 x 11 tiles of 384 threads, two CTAs (24 warps) per SM at 80 registers (about 500 bytes of spills a
// thread, which the L1 beside 88 KB of shared memory a tile mostly holds): the tile's 747 faces are
// two rounds of 384 threads (97 % of them busy).  Four steps of 1024^2 / one of the wind: 1.89 / 3.30 ms;
// 32 x 8 with 256 threads, three CTAs 2.10 / 3.42; 32 x 9 with 320 threads at 96 registers 2.04 / 3.45;
// 32 x 8 with 288 at 112 registers 2.24 / 3.66 (those where this took 1.92 / 3.35).  One HLLD step at 1024^2: 0.42 ms, 0.98 in FP64, 0.37 with one
// set of units for the tile.
constexpr int kTY = 11;
constexpr int kTYDual = 8;

template <int ORDER, int NT>
void launch_tiles(const Params& P, dim3 grid, const CPlanes& in, const Planes& out,
                  const double* T_do, unsigned long long* T_bits, Scalars* rot, Scalars* ctr,
                  int dt_only, cudaStream_t st, double* aux) {
    constexpr size_t n = ShapeInt<ORDER, kTY>::bytes;
    if (P.method == GD_METHOD_HLLD)
        mhd_fast_kernel<ORDER, kTY, true, NT><<<grid, NT, n, st>>>(P, in, out, T_do, T_bits, rot,
                                                                   ctr, dt_only, aux);
    else
        mhd_fast_kernel<ORDER, kTY, false, NT><<<grid, NT, n, st>>>(P, in, out, T_do, T_bits, rot,
                                                                    ctr, dt_only, aux);
}

template <int ORDER>
cudaError_t launch_t(const Params& P, const CPlanes& in, const Planes& out, const double* T_do,
                     unsigned long long* T_bits, Scalars* rot, Scalars* ctr, int dt_only,
                     cudaStream_t st, double* aux = nullptr) {
    const dim3 grid((P.N + TX - 1) / TX, P.tile_rows ? P.tile_rows : (P.M + kTY - 1) / kTY);
    if ((long long)grid.x * grid.y <= P.few_tiles)
        launch_tiles<ORDER, kNTFew>(P, grid, in, out, T_do, T_bits, rot, ctr, dt_only, st, aux);
    else
        launch_tiles<ORDER, kNT>(P, grid, in, out, T_do, T_bits, rot, ctr, dt_only, st, aux);
    return cudaGetLastError();
}

template <int ORDER>
cudaError_t launch_tangent_t(const Params& P, const CPlanes& in, const CPlanes& din,
                             const Planes& dout, const double* T_do, cudaStream_t st) {
    dim3 grid((P.N + TX - 1) / TX, (P.M + kTYDual - 1) / kTYDual);
    mhd_tangent_kernel<ORDER, kTYDual><<<grid, NTDual, SmemM<Dual, ORDER, kTYDual>::bytes, st>>>(
        P, in, din, dout, T_do);
    return cudaGetLastError();
}

template <int ORDER, bool HLLD>
cudaError_t set_room() {
    constexpr int n = (int)ShapeInt<ORDER, kTY>::bytes;
    constexpr auto what = cudaFuncAttributeMaxDynamicSharedMemorySize;
    cudaError_t e = cudaFuncSetAttribute(mhd_fast_kernel<ORDER, kTY, HLLD, kNT>, what, n);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(mhd_fast_kernel<ORDER, kTY, HLLD, kNTFew>, what, n);
    return e;
}

}  // namespace

int mhd_tile_height() { return kTY; }

cudaError_t prepare_mhd_fast() {
    cudaError_t e = set_room<1, true>();
    if (e == cudaSuccess) e = set_room<1, false>();
    if (e == cudaSuccess) e = set_room<2, true>();
    if (e == cudaSuccess) e = set_room<2, false>();
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(mhd_tangent_kernel<1, kTYDual>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)SmemM<Dual, 1, kTYDual>::bytes);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(mhd_tangent_kernel<2, kTYDual>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)SmemM<Dual, 2, kTYDual>::bytes);
    return e;
}

cudaError_t launch_mhd_fast(const Params& P, const CPlanes& in, const Planes& out,
                            const double* T_do, unsigned long long* T_bits, Scalars* rot,
                            Scalars* ctr, int dt_only, cudaStream_t st) {
    if (P.order == 1) return launch_t<1>(P, in, out, T_do, T_bits, rot, ctr, dt_only, st);
    return launch_t<2>(P, in, out, T_do, T_bits, rot, ctr, dt_only, st);
}

cudaError_t launch_mhd_fast_aux(const Params& P, const CPlanes& in, const Planes& out,
                                const double* T_do, unsigned long long* T_bits, Scalars* rot,
                                Scalars* ctr, double* aux, cudaStream_t st) {
    if (P.order == 1) return launch_t<1>(P, in, out, T_do, T_bits, rot, ctr, 0, st, aux);
    return launch_t<2>(P, in, out, T_do, T_bits, rot, ctr, 0, st, aux);
}

cudaError_t launch_mhd_tangent(const Params& P, const CPlanes& in, const CPlanes& din,
                               const Planes& dout, const double* T_do, cudaStream_t st) {
    if (P.order == 1) return launch_tangent_t<1>(P, in, din, dout, T_do, st);
    return launch_tangent_t<2>(P, in, din, dout, T_do, st);
}


namespace {
// One face per thread through the step's own face solver (side + hlld_local): L, R are n x 8
// in the reference's HLLDQ_Korolkov layout (rho, p, vx, vy, vz, Bx, By, Bz; Gaussian B, vz
// taken as 0 as the 2-D step does); flux n x 8 in its output order and units (mass, x, y, z
// momentum, Bx, By, Bz, energy; the z-momentum flux is not formed by the 2-D step: 0);
// speed n values max(|S_L|, |S_R|).  The field goes to Heaviside-Lorentz units by the
// rounded product the tile load uses.  axis 0: normal +x.
__global__ void mhd_face_probe_kernel(Params P, long long n, int axis,
                                      const double* __restrict__ L,
                                      const double* __restrict__ R, double* flux,
                                      double* speed) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double* a = L + 8 * i;
    const double* b = R + 8 * i;
    const bool isx = axis == 0;
    double qa[NF], qb[NF];
    qa[0] = a[0]; qa[1] = a[1]; qa[2] = a[2]; qa[3] = a[3];
    qb[0] = b[0]; qb[1] = b[1]; qb[2] = b[2]; qb[3] = b[3];
#pragma unroll
    for (int f = 4; f < NF; ++f) {
        qa[f] = __dmul_rn(a[f + 1], kInvSpi4);
        qb[f] = __dmul_rn(b[f + 1], kInvSpi4);
    }
    double la[NF], lb[NF];  // in the face's frame
#pragma unroll
    for (int f = 0; f < NF; ++f) {
        const int g = isx || f < 2 || f == 6 ? f : (f < 4 ? 5 - f : 9 - f);
        la[f] = qa[g];
        lb[f] = qb[g];
    }
    double UU;
    fx::FluxI G;
    FluxM<double> F;
    if (P.method == GD_METHOD_HLLD ? fx::mhd_face<true>(la, lb, P.gas, G, UU)
                                   : fx::mhd_face<false>(la, lb, P.gas, G, UU))
        F = FluxM<double>{G.m, G.mn, G.mt, G.e, G.bn, G.bt, G.bz};
    else
        F = float_flux_of(P, la, lb, UU);
    double* o = flux + 8 * i;
    o[0] = F.m;
    o[1] = isx ? F.mn : F.mt;
    o[2] = isx ? F.mt : F.mn;
    o[3] = 0.0;
    o[4] = (isx ? F.bn : F.bt) * kSpi4;
    o[5] = (isx ? F.bt : F.bn) * kSpi4;
    o[6] = F.bz * kSpi4;
    o[7] = F.e;
    speed[i] = dabs(UU);
}
}  // namespace

cudaError_t launch_mhd_face_probe(const Params& P, long long n, int axis, const double* L,
                                  const double* R, double* flux, double* speed,
                                  cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    const long long blocks = (n + 255) / 256;
    mhd_face_probe_kernel<<<(unsigned int)blocks, 256, 0, st>>>(P, n, axis, L, R, flux, speed);
    return cudaGetLastError();
}

}  // namespace gd
