// gd_fast_euler.cu -- fused minmod-TVD + HLLC/HLL + update step for 2-D Euler, face-once tiles.
//
// One CTA owns a TX x TY tile.  Phases, separated by __syncthreads():
//   L  load the tile plus a 2-cell cross-shaped halo (boundary ghosts applied) into smem;
//   S  per-cell minmod slopes along x and y (integer-pipe minmod, one FP64 sub per edge);
//   F  every face of the tile once: left/right face states from the slopes, the HLLC (or,
//      for method 0, HLL) flux in the face's local (normal, tangent) frame, and the face's
//      wave-speed maximum;
//   U  conservative update of each cell from its four face fluxes, positivity floors,
//      primitive recovery; store; block dt minimum and the fused funk_time rotation.
// The reference computes every face twice, once from each neighbour (kernel.cu:3560-3586);
// here each face is computed once and used with opposite signs by its two cells.
//
// S and F of the step run in scaled 64-bit integers (gd_fixed.cuh): a tile's cells are held as
// significands and exponents, each face takes powers of two over its own stencil as units, slopes
// and face states are integer adds, the flux an integer chain; only the flux results and the update
// are FP64.  A face whose densities' or pressures' exponents span more than 8, or whose fan leaves
// the integers' range, is solved in FP64 from the cells themselves.  The tangent's tile (Dual) is
// floating point throughout: its standalone products run on the integer pipes (mulx: the FP64
// multiply's bits), the sound speeds and reciprocals take two FP64 operations each, and the HLLC
// star state takes S_M and q from one reciprocal.
//
// A face's arithmetic depends on its stencil alone and every operation of the update is written
// out, so that tile shapes, thread counts and kernels agree bit for bit.
//
// Two kernels share the tile body: euler_fast_kernel (one grid, one CTA per tile) and
// euler_batch_kernel (a persistent launch that walks the tiles of many independent grids,
// each grid with its own parameters, state, dt reduction and funk_time rotation).  Tile
// shapes 16x16, 32x8, 32x16 and 64x8 are compiled; the autotuner picks one for a batch, and
// the single-grid step uses 16x16 (64 registers a thread: four CTAs, 32 warps, per SM).
//
// Reference semantics kept: primitive reconstruction of (rho, p, vx, vy) with the rho/p
// face fallback to the cell value (kernel.cu:3436-3544), Davis wave speeds and the HLLC
// star states of HLLC_Aleksashov (kernel.cu:853-1165), the HLL flux (kernel.cu:1485-1609)
// for method 0, the Ker_Dekard update and floors
// rho <= 0 -> 1e-4, p <= 0 -> 1e-6 (kernel.cu:1849-1874), dt = min over faces of
// krit*rad/max(|SL|,|SR|) with rad = dy on x-faces (kernel.cu:1811).
#include <type_traits>

#include "gd_dual.cuh"
#include "gd_internal.cuh"
#include "gd_kernels.h"
#include "gd_mhd_flux.cuh"  // cst<T>

namespace gd {
namespace {

constexpr int kNT = 256;  // threads of a tile: single-grid step
// The tangent's 552 faces in two rounds: 20 tangent steps at 512^2 take 4.73 ms, 4.95 with 256
// threads, 5.30 with 384.
constexpr int kNTTan = 288;
// Threads of a tile of the 16x16 shape where every tile has an SM to itself (Params::few_tiles): the
// step is then one tile's latency, and 576 threads take its 544 faces in one round instead of
// three: 11.4 against 13.9 us at 64x48, 12.1 against 14.3 at 192x192 (144 tiles).  From two
// tiles on an SM (156 tiles: 19.0 against 16.1 us) the 256-thread tiles share
// an SM better.  The threads of a tile change no result: faces and cells are independent.
constexpr int kNTFew = 576;
constexpr int NF = 4;
// CTAs per SM that the shared memory of a tile shape leaves room for
template <int TX, int TY>
constexpr int kCtas = TX * TY > 256 ? 2 : 4;
// threads of a tile in the batch kernel (see there)
template <int TX, int TY>
constexpr int kNTBatch = TX * TY > 256 ? 256 : 192;

template <class T>
struct FluxE {
    T m, mn, mt, e;
};

// HLLC flux in a local frame: un = normal velocity, ut = in-plane tangential velocity.
// Returns the flux (mass, normal momentum, tangential momentum, energy) and, in UU, SL or
// SR, the one of larger magnitude (signed; the dt reduction takes |UU|).  T is double, or
// Dual for the tangent (value and derivative, the branch choices taken on the value).
// Products go through mulx (on the integer pipes for double), sums and fused
// multiply-adds through the FP64 unit.
template <class T>
__device__ __forceinline__ FluxE<T> hllc_local(T rL, T pL, T unL, T utL, T rR, T pR, T unR,
                                               T utR, const Params& P, T& UU) {
    const double g = P.gamma;
    const T cL = sqrt_over_2op(mulx(g, pL), rL);  // sqrt(g p / rho)
    const T cR = sqrt_over_2op(mulx(g, pR), rR);
    const T aL = unL - cL, aR = unR - cR;
    const T bL = unL + cL, bR = unR + cR;
    const T SL = dmin(aL, aR);  // Davis estimates (kernel.cu:981-982)
    const T SR = dmax(bL, bR);
    const T suL = SL - unL, suR = SR - unR;
    const T mL = mulx(rL, suL), mR = mulx(rR, suR);
    // S_M = Nm / D (kernel.cu:1001-1003): its sign is the sign of Nm times that of D
    const T Nm = fma(mR, unR, fma(-mL, unL, pL - pR));
    const T D = mR - mL;
    UU = max_nonneg(SL, SR);  // signed: the block reduction takes the magnitude

    // Side whose state (or star state) gives the flux at x/t = 0 (kernel.cu:1119-1158).
    const bool takeL = gt_zero(SL) || !quotient_neg(Nm, D);
    const T r = takeL ? rL : rR;
    const T p = takeL ? pL : pR;
    const T un = takeL ? unL : unR;
    const T ut = takeL ? utL : utR;
    const T S = takeL ? SL : SR;
    const T su = takeL ? suL : suR;
    const T mm = takeL ? mL : mR;
    const bool star = takeL ? !gt_zero(SL) : ge_zero(SR);

    const T V2 = fma(un, un, mulx(ut, ut));
    FluxE<T> F;
    if (star) {
        // F_K + S_K (U*_K - U_K) is the physical flux of the star state, F(U*_K) with the
        // star pressure: the jump conditions across S_K are what define rho*, p* and E*
        // (kernel.cu:1119-1158).  With q = S_M / (S_K - S_M), p* = p + rho su (S_M - un),
        // su = S_K - un and G = gamma / (gamma - 1):
        //   mass rho* S_M = rho su q,  momentum rho* S_M^2 + p*,  tangential rho* S_M ut,
        //   energy (E* + p*) S_M = q su (p G + rho (|v|^2 / 2 + S_K (S_M - un))).
        // S_M and q from one reciprocal: with X = S_K D - Nm = D (S_K - S_M),
        //   S_M = Nm X / (D X),  q = Nm D / (D X).
        const T X = fma(S, D, -Nm);
        const T R = rcp_2op(mulx(D, X));
        const T NR = mulx(Nm, R);
        const T SM = mulx(NR, X);
        const T q = mulx(NR, D);
        const T SMu = SM - un;
        const T pst = fma(mm, SMu, p);
        const T qs = mulx(q, su);
        F.m = mulx(r, qs);
        F.mn = fma(F.m, SM, pst);
        F.mt = mulx(F.m, ut);
        F.e = mulx(qs, fma(p, P.g_gm1, mulx(r, fma(0.5, V2, mulx(S, SMu)))));
    } else {
        F.m = mulx(r, un);
        F.mn = fma(F.m, un, p);
        F.mt = mulx(F.m, ut);
        F.e = mulx(un, fma(p, P.g_gm1, mulx(mulx(0.5, r), V2)));  // (E + p) un
    }
    return F;
}

// HLL flux of kernel.cu:1485-1609 in a local frame (same arguments and results as
// hllc_local): sound speed 0 where rho <= 0, D_L = min(un) - max(c), D_R = max(un) + max(c),
// the upwind physical flux when the fan lies on one side of the face (strict tests against
// Omega = 0, kernel.cu:11), else (D_R F_L - D_L F_R + D_L D_R (U_R - U_L)) / (D_R - D_L).
// Its products stay on the FP64 unit: the tile function holds both fluxes, and registers
// are allocated for its heavier path -- integer-pipe products here took the tile to about
// 110 registers a thread, two CTAs per SM for the HLLC step as well.
template <class T>
__device__ __forceinline__ FluxE<T> hll_local(T rL, T pL, T unL, T utL, T rR, T pR, T unR,
                                              T utR, const Params& P, T& UU) {
    const double g = P.gamma;
    const T gpL = g * pL, gpR = g * pR;
    const T cL = le_zero(rL) ? cst<T>(0.0) : sqrt_over(gpL, rL);  // sqrt(g p / rho)
    const T cR = le_zero(rR) ? cst<T>(0.0) : sqrt_over(gpR, rR);
    const T cm = max_nonneg(cL, cR);
    const T DL = dmin(unL, unR) - cm;
    const T DR = dmax(unL, unR) + cm;
    UU = max_nonneg(DL, DR);  // signed: the block reduction takes the magnitude
    const bool left = gt_zero(DL), right = !left && lt_zero(DR);
    FluxE<T> F;
    if (left || right) {  // one side's physical flux
        const T r = left ? rL : rR, p = left ? pL : pR;
        const T un = left ? unL : unR, ut = left ? utL : utR;
        F.m = r * un;
        F.mn = fma(F.m, un, p);
        F.mt = F.m * ut;
        const T E = fma(p, P.inv_gm1, 0.5 * r * fma(un, un, ut * ut));
        F.e = (E + p) * un;
        return F;
    }
    const T mL = rL * unL, mR = rR * unR;
    const T EL = fma(pL, P.inv_gm1, 0.5 * rL * fma(unL, unL, utL * utL));
    const T ER = fma(pR, P.inv_gm1, 0.5 * rR * fma(unR, unR, utR * utR));
    const T inv = rcp_fast(DR - DL);
    const T dd = DL * DR;
    // (D_R F_L - D_L F_R + D_L D_R dU) / (D_R - D_L), component by component
    F.m = fma(dd, rR - rL, fma(DR, mL, -DL * mR)) * inv;
    F.mn = fma(dd, mR - mL, fma(DR, fma(mL, unL, pL), -DL * fma(mR, unR, pR))) * inv;
    F.mt = fma(dd, fma(rR, utR, -rL * utL), fma(DR, mL * utL, -DL * (mR * utR))) * inv;
    F.e = fma(dd, ER - EL, fma(DR, (EL + pL) * unL, -DL * ((ER + pR) * unR))) * inv;
    return F;
}

template <int ORDER, int TX, int TY>
struct Shape {
    static constexpr int H = ORDER == 2 ? 2 : 1;
    static constexpr int SX = TX + 2 * H;
    static constexpr int SY = TY + 2 * H;
    static constexpr int kPrim = NF * SY * SX;
    static constexpr int kSlx = ORDER == 2 ? NF * TY * (TX + 2) : 0;
    static constexpr int kSly = ORDER == 2 ? NF * (TY + 2) * TX : 0;
    static constexpr int kFx = NF * TY * (TX + 1);
    static constexpr int kFy = NF * (TY + 1) * TX;
    static constexpr int kKey = SY * SX;
    static constexpr int kCell = NF * TY * TX;
    static constexpr size_t bytes = sizeof(double) * (kKey + kPrim + kCell + kFx + kFy);
    static constexpr size_t dual_bytes = 2 * sizeof(double) * (kPrim + kSlx + kSly + kFx + kFy);
};

// Value and tangent planes (the tangent step of the adjoint checks).
struct DualIn {
    CPlanes v, d;
};
struct DualOut {  // the tangent alone: the values are the recorded run's
    Planes d;
};

__device__ __forceinline__ void load_cell(const Params& P, const CPlanes& in, int gx, int gy,
                                          double* v) {
    fetch_cell<NF>(P, in, gx, gy, v);
}
// The tangent of a ghost value: the same copy (the tangent runs on periodic grids only, where
// a ghost is a copy of a cell).
__device__ __forceinline__ void load_cell(const Params& P, const DualIn& in, int gx, int gy,
                                          Dual* v) {
    double a[NF], b[NF];
    fetch_cell<NF>(P, in.v, gx, gy, a);
    fetch_cell<NF>(P, in.d, gx, gy, b);
#pragma unroll
    for (int f = 0; f < NF; ++f) v[f] = Dual{a[f], b[f]};
}
__device__ __forceinline__ void store_cell(const Planes& out, long long k, int f, double x) {
    store_f(out, f, k, x);
}
__device__ __forceinline__ void store_cell2(const Planes& out, long long k, int f0, double a,
                                            double b) {
    store_pair(out, f0, k, a, b);
}
__device__ __forceinline__ void store_cell(const DualOut& out, long long k, int f, Dual x);
__device__ __forceinline__ void store_cell2(const DualOut& out, long long k, int f0, Dual a,
                                            Dual b) {
    store_cell(out, k, f0, a);
    store_cell(out, k, f0 + 1, b);
}
__device__ __forceinline__ void store_cell(const DualOut& out, long long k, int f, Dual x) {
    out.d.f[f][k] = x.d;
}

// The arrays of a tile in shared memory.
template <class T, int ORDER, int TX, int TY>
struct TileMem {
    using S = Shape<ORDER, TX, TY>;
    T *prim;  // [NF][SY][SX]
    T *slx;   // [NF][TY][TX+2]   cells x in [-1, TX]
    T *sly;   // [NF][TY+2][TX]   cells y in [-1, TY]
    T *fx;    // [NF][TY][TX+1]   face between x-1 and x
    T *fy;    // [NF][TY+1][TX]   face between y-1 and y
    __device__ explicit TileMem(T* smem)
        : prim(smem), slx(prim + S::kPrim), sly(slx + S::kSlx), fx(sly + S::kSly),
          fy(fx + S::kFx) {}
};
// The step's: the cells' significands and keys (gd_fixed.cuh), and the tile's own values.
template <int ORDER, int TX, int TY>
struct TileMemInt {
    using S = Shape<ORDER, TX, TY>;
    using Key = fx::Keys<NF>;
    static_assert(sizeof(Key) == sizeof(double), "keys take one double a cell");
    Key* key;      // [SY][SX]
    fx::i64* q;    // [NF][SY][SX]
    double* cell;  // [NF][TY][TX]
    double *fx, *fy;
    __device__ explicit TileMemInt(double* smem)
        : key(reinterpret_cast<Key*>(smem)), q(reinterpret_cast<fx::i64*>(smem + S::kKey)),
          cell(smem + S::kKey + S::kPrim), fx(cell + S::kCell), fy(fx + S::kFx) {}
};

// One face of a tile: faces 0 .. NFX-1 have an x normal, the rest a y normal.
template <int TX, int TY>
struct Face {
    static constexpr int NFX = (TX + 1) * TY, NFY = TX * (TY + 1), kAll = NFX + NFY;
    bool isx, used;
    int lx, ly;
    // used: inside the grid, and next to a cell that the step updates
    __device__ Face(const Params& P, int tx0, int ty0, int i) {
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
    template <class T>
    __device__ __forceinline__ void store(T* fx, T* fy, T m, T e, T mn, T mt) const {
        if (isx) {
            T* fo = fx + ly * (TX + 1) + lx;
            fo[0 * TY * (TX + 1)] = m;
            fo[1 * TY * (TX + 1)] = e;
            fo[2 * TY * (TX + 1)] = mn;  // x momentum
            fo[3 * TY * (TX + 1)] = mt;  // y momentum
        } else {
            T* fo = fy + ly * TX + lx;
            fo[0 * (TY + 1) * TX] = m;
            fo[1 * (TY + 1) * TX] = e;
            fo[2 * (TY + 1) * TX] = mt;  // x momentum
            fo[3 * (TY + 1) * TX] = mn;  // y momentum
        }
    }
};

// The flux in floating point between the states qa (low side) and qb, {rho, p, normal,
// tangential velocity}, with the solver of the step's method.
template <class T>
__device__ __forceinline__ FluxE<T> flux_of(const Params& P, const T* qa, const T* qb, T& UU) {
    return P.method == GD_METHOD_HLL
               ? hll_local(qa[0], qa[1], qa[2], qa[3], qb[0], qb[1], qb[2], qb[3], P, UU)
               : hllc_local(qa[0], qa[1], qa[2], qa[3], qb[0], qb[1], qb[2], qb[3], P, UU);
}
// The states on either side of a face, c + d/2 and c - d/2; rho and p fall back to the cell
// value (kernel.cu:3436-3470).
template <class T>
__device__ __forceinline__ void side_states(int f, T ca, T da, T cb, T db, T& a, T& b) {
    a = fma(0.5, da, ca);
    b = fma(-0.5, db, cb);
    if (f < 2) {
        a = le_zero(a) ? ca : a;
        b = le_zero(b) ? cb : b;
    }
}

template <class T, int ORDER, int TX, int TY>
__device__ __forceinline__ T face_flux(const Params& P, const TileMem<T, ORDER, TX, TY>& t,
                                       const Face<TX, TY>& w) {
    using S = Shape<ORDER, TX, TY>;
    constexpr int H = S::H, SX = S::SX, SY = S::SY;
    const int lx = w.lx, ly = w.ly;
    const T* pb = t.prim + (ly + H) * SX + (lx + H);
    const T* pa = pb - (w.isx ? 1 : SX);
    T qa[NF], qb[NF], UU;
#pragma unroll
    for (int f = 0; f < NF; ++f) {
        const int g = f < 2 ? f : (w.isx ? f : 5 - f);  // field of the local frame's component f
        qa[f] = pa[g * SY * SX];
        qb[f] = pb[g * SY * SX];
        if (ORDER == 2) {
            T da, db;
            if (w.isx) {
                da = t.slx[(g * TY + ly) * (TX + 2) + lx];
                db = t.slx[(g * TY + ly) * (TX + 2) + lx + 1];
            } else {
                da = t.sly[(g * (TY + 2) + ly) * TX + lx];
                db = t.sly[(g * (TY + 2) + ly + 1) * TX + lx];
            }
            side_states(f, qa[f], da, qb[f], db, qa[f], qb[f]);
        }
    }
    const FluxE<T> F = flux_of(P, qa, qb, UU);
    w.store(t.fx, t.fy, F.m, F.e, F.mn, F.mt);
    return UU;
}

struct Speeds {
    double x, y;
    __device__ __forceinline__ void take(bool isx, double UU) {
        if (isx) x = max_nonneg(x, UU);
        else y = max_nonneg(y, UU);
    }
};

struct TileResult {
    double umax_x, umax_y;
    bool any_active;
    unsigned int nfl_r, nfl_p, nbad;
};

// a b rounded by itself: every operation of the update is written out, so that the kernels that
// inline it round alike whatever the compiler would contract in each.
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ Dual mul_rn(Dual a, Dual b) { return a * b; }
__device__ __forceinline__ Dual mul_rn(double a, Dual b) { return a * b; }

// ---- U: conservative update of the tile's cells ---------------------------------------------
// cell: the tile's own values, rows RS and fields FS apart.
template <class T, int ORDER, int TX, int TY, int NT, int RS, int FS, class OUT>
__device__ __forceinline__ void update_cells(const Params& P, const OUT& out, int tx0, int ty0,
                                             double T_do, int dt_only, const T* cell, const T* fx,
                                             const T* fy, TileResult& res, double* aux) {
    const int N = P.N, M = P.M;
    const double kx = T_do * P.inv_dx, ky = T_do * P.inv_dy;
    bool any_active = false;
    unsigned int nfl_r = 0, nfl_p = 0, nbad = 0;
    for (int i = threadIdx.x; i < TX * TY; i += NT) {
        const int ly = i / TX, lx = i - ly * TX;
        const int gx = tx0 + lx, gy = ty0 + ly;
        if (gx >= N || gy >= M) continue;
        const T* c = cell + ly * RS + lx;
        const T r = c[0], p = c[FS], u = c[2 * FS], v = c[3 * FS];
        const long long k = (long long)gy * N + gx;
        if (P.frozen && !cell_active(P, gx, gy)) {  // the faces' own test
            if (!dt_only) {
                store_cell2(out, k, 0, r, p);
                store_cell2(out, k, 2, u, v);
            }
            continue;
        }
        any_active = true;
        if (dt_only) continue;
        const T* fxc = fx + ly * (TX + 1) + lx;
        const T* fyc = fy + ly * TX + lx;
        T d[NF];
#pragma unroll
        for (int f = 0; f < NF; ++f) {
            const T* a = fxc + f * TY * (TX + 1);
            const T* b = fyc + f * (TY + 1) * TX;
            d[f] = fma(kx, a[1] - a[0], mul_rn(ky, b[TX] - b[0]));
        }
        if constexpr (std::is_same<T, double>::value) {
            if (aux != nullptr) {  // the recording of the adjoint: the flux differences used
                const long long KK = (long long)N * M;
#pragma unroll
                for (int f = 0; f < NF; ++f) aux[f * KK + k] = d[f];
            }
        }
        T r2 = r - d[0];
        if (le_zero(r2)) { r2 = cst<T>(0.0001); ++nfl_r; }
        const T inv = rcp_fast(r2);
        const T mx2 = fma(r, u, -d[2]), my2 = fma(r, v, -d[3]);
        const T u2 = mul_rn(mx2, inv);
        const T v2 = mul_rn(my2, inv);
        // p' = (gamma - 1) (E - d_E - K'/2) with E = p / (gamma - 1) + K / 2, K = rho |v|^2,
        // K' = rho' |v'|^2 = m' . v' (kernel.cu:1861-1870)
        const T K2 = fma(mx2, u2, mul_rn(my2, v2));
        const T dK = fma(r, fma(u, u, mul_rn(v, v)), -K2);
        T p2 = fma(P.hgm1, dK, fma(-P.gm1, d[1], p));
        if (le_zero(p2)) { p2 = cst<T>(0.000001); ++nfl_p; }
        if (!finite_bits(r2) || !finite_bits(p2) || !finite_bits(u2) || !finite_bits(v2)) ++nbad;
        store_cell2(out, k, 0, r2, p2);
        store_cell2(out, k, 2, u2, v2);
    }
    res.any_active = any_active;
    res.nfl_r = nfl_r;
    res.nfl_p = nfl_p;
    res.nbad = nbad;
}

// The tangent's tile: slopes in shared memory, faces in floating point on Dual values.
template <class T, int ORDER, int TX, int TY, int NT, class IN, class OUT>
__device__ __noinline__ void euler_tile(const Params& P, const IN& in, const OUT& out, int tx0,
                                        int ty0, double T_do, int dt_only, T* smem,
                                        TileResult& res, double* aux) {
    using S = Shape<ORDER, TX, TY>;
    constexpr int H = S::H, SX = S::SX, SY = S::SY;
    const TileMem<T, ORDER, TX, TY> mem(smem);
    T *prim = mem.prim, *slx = mem.slx, *sly = mem.sly, *fx = mem.fx, *fy = mem.fy;

    const int tid = threadIdx.x;
    const int N = P.N, M = P.M;

    // ---- L: tile + cross halo ------------------------------------------------------------
    for (int i = tid; i < SY * SX; i += NT) {
        const int ly = i / SX, lx = i - ly * SX;
        const bool xh = lx < H || lx >= TX + H, yh = ly < H || ly >= TY + H;
        if (xh && yh) continue;  // corners are never read
        const int gx = tx0 + lx - H, gy = ty0 + ly - H;
        T v[NF];
        if (gx >= -2 && gx < N + 2 && gy >= -2 && gy < M + 2 &&
            !((gx < 0 || gx >= N) && (gy < 0 || gy >= M))) {
            load_cell(P, in, gx, gy, v);
        } else {
#pragma unroll
            for (int f = 0; f < NF; ++f) v[f] = cst<T>(1.0);  // outside the grid, never used
        }
#pragma unroll
        for (int f = 0; f < NF; ++f) prim[(f * SY + ly) * SX + lx] = v[f];
    }
    __syncthreads();

    // ---- S: slopes --------------------------------------------------------------------------
    // A thread takes a run of G cells along the direction, so neighbouring slopes share their
    // difference: G + 1 FP64 subtractions per G cells instead of 2 G.
    if (ORDER == 2) {
        constexpr int GX = (TX + 2) % 3 == 0 ? 3 : 2, GY = (TY + 2) % 3 == 0 ? 3 : 2;
        constexpr int NGX = (TX + 2) / GX, NGY = (TY + 2) / GY;
        static_assert((TX + 2) % GX == 0 && (TY + 2) % GY == 0, "slope runs tile the rows");
        for (int i = tid; i < TY * NGX; i += NT) {
            const int ly = i / NGX, c0 = (i - ly * NGX) * GX;  // cells x = c0 - 1 ...
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
        for (int i = tid; i < NGY * TX; i += NT) {
            const int g = i / TX, lx = i - g * TX, r0 = g * GY;  // cells y = r0 - 1 ...
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

    // ---- F: faces ---------------------------------------------------------------------------
    Speeds fastest{0.0, 0.0};
    for (int i = tid; i < Face<TX, TY>::kAll; i += NT) {
        const Face<TX, TY> f(P, tx0, ty0, i);
        if (f.used) fastest.take(f.isx, value_of(face_flux<T, ORDER, TX, TY>(P, mem, f)));
    }
    __syncthreads();

    update_cells<T, ORDER, TX, TY, NT, SX, SY * SX>(P, out, tx0, ty0, T_do, dt_only,
                                                prim + H * SX + H, fx, fy, res, aux);
    res.umax_x = fastest.x;
    res.umax_y = fastest.y;
}

// ---- The step's tile: face work in 64-bit integers --------------------------------------------
//
// The cells of the tile and its halo are held as significands and exponents (gd_fixed.cuh); a face
// shifts its stencil to units of its own.  Slopes, minmod and face states are then plain 64-bit
// adds and selects, and the HLLC flux is fx::hllc: the FP64 pipe is left with the conversion of
// the fluxes and the update (about 44 instructions a cell instead of 103).  Bound by the ALU (69 %),
// FP64 (63 %) and the chains between (issue 63 %): one step at 4096^2 takes 1.86 ms, 3.86 in FP64, 1.70
// with one set of units for the tile, which cut small components (see face_states).

// One compiled body for every kernel, so that a face left to floating point has the same bits
// whichever kernel solves it.
__device__ __noinline__ FluxE<double> float_flux(const Params& P, const double* qa,
                                                 const double* qb, double& UU) {
    return flux_of(P, qa, qb, UU);
}

// The faces that the integer solver left, in floating point from the cells themselves.  Out of
// line, and after the loop over the faces: a second solver inside it would take registers from
// every face for what a few need; and as a list for the whole block, so that a few faces of each
// warp cost what they are (a step of 1024^2 cells with densities and pressures at random over 2^6:
// 239 us, 489 with each thread redoing its own).
template <int ORDER, int TX, int TY, int NT>
__device__ __noinline__ void faces_left(const Params& P, const CPlanes& in, double* smem, int tx0,
                                        int ty0, const LeftFaces<Face<TX, TY>::kAll>& left,
                                        Speeds& u) {
    const TileMemInt<ORDER, TX, TY> t(smem);
    for (unsigned int k = threadIdx.x; k < left.n; k += NT) {
        const Face<TX, TY> w(P, tx0, ty0, left.face(k));
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
            qa[f] = c[1][f];
            qb[f] = c[2][f];
            if (ORDER == 2) {
                const double d = qb[f] - qa[f];
                side_states(f, qa[f], minmod(qa[f] - c[0][f], d), qb[f],
                            minmod(d, c[3][f] - qb[f]), qa[f], qb[f]);
            }
        }
        const double la[NF] = {qa[0], qa[1], w.isx ? qa[2] : qa[3], w.isx ? qa[3] : qa[2]};
        const double lb[NF] = {qb[0], qb[1], w.isx ? qb[2] : qb[3], w.isx ? qb[3] : qb[2]};
        const FluxE<double> F = float_flux(P, la, lb, UU);
        w.store(t.fx, t.fy, F.m, F.e, F.mn, F.mt);
        if (left.no_speed(k)) u.take(w.isx, UU);
    }
}

// Every face of a tile, up to those left.  dt_only: the wave speeds alone.
template <bool HLL, int ORDER, int TX, int TY, int NT>
__device__ __forceinline__ void faces(const Params& P, double* smem, int tx0, int ty0, int dt_only,
                                      LeftFaces<Face<TX, TY>::kAll>& left, Speeds& u) {
    using S = Shape<ORDER, TX, TY>;
    using fx::i64;
    const TileMemInt<ORDER, TX, TY> t(smem);
    for (int i = threadIdx.x; i < Face<TX, TY>::kAll; i += NT) {
        const Face<TX, TY> w(P, tx0, ty0, i);
        if (!w.used) continue;
        const int c = (w.ly + S::H) * S::SX + w.lx + S::H, st = w.isx ? 1 : S::SX;
        i64 a[NF], b[NF];
        int top[NF];
        double F[NF], UU;
        bool speed_ok = false, done = false;
        if (P.gas.room >= 0 && fx::face_states<NF, ORDER>(t.q + c, st, S::SY * S::SX, t.key + c, st,
                                                          w.isx, a, b, top))
            done = fx::euler_flux<HLL>(a, b, top, P.gas, F, UU, speed_ok, dt_only);
        if (speed_ok) u.take(w.isx, UU);
        if (!done) left.add(i, speed_ok);
        else if (!dt_only) w.store(t.fx, t.fy, F[0], F[3], F[1], F[2]);
    }
}

// One TX x TY tile of the step whose lower-left cell is (tx0, ty0).  Reads `in`, writes `out`,
// returns the per-thread wave-speed maxima and counters.  Every thread of the block must call it.
// `aux` (may be null): per cell, the flux differences d[0..3] of the update, planes of N*M
// (the adjoint's recording).  METHODS: 1 HLLC, 2 HLL, 3 the one of P (both solvers in the
// function).
template <int METHODS, int ORDER, int TX, int TY, int NT>
__device__ __forceinline__ void step_tile(const Params& P, const CPlanes& in, const Planes& out,
                                          int tx0, int ty0, double T_do, int dt_only,
                                          double* smem, TileResult& res, double* aux) {
    using S = Shape<ORDER, TX, TY>;
    constexpr int H = S::H, SX = S::SX, SY = S::SY;
    const TileMemInt<ORDER, TX, TY> t(smem);
    __shared__ LeftFaces<Face<TX, TY>::kAll> left;
    if (threadIdx.x == 0) left.n = 0;
    const int N = P.N, M = P.M;
    for (int i = threadIdx.x; i < SY * SX; i += NT) {
        const int ly = i / SX, lx = i - ly * SX;
        const bool xh = lx < H || lx >= TX + H, yh = ly < H || ly >= TY + H;
        const int gx = tx0 + lx - H, gy = ty0 + ly - H;
        if ((xh && yh) || gx < -2 || gx >= N + 2 || gy < -2 || gy >= M + 2 ||
            ((gx < 0 || gx >= N) && (gy < 0 || gy >= M)))
            continue;  // no face reads it
        double v[NF];
        load_cell(P, in, gx, gy, v);
        fx::cell_units<NF>(v, t.q + i, SY * SX, t.key[i]);
        if (!xh && !yh) {
#pragma unroll
            for (int f = 0; f < NF; ++f) t.cell[(f * TY + ly - H) * TX + lx - H] = v[f];
        }
    }
    __syncthreads();
    Speeds fastest{0.0, 0.0};
    if (METHODS == 2 || (METHODS == 3 && P.method == GD_METHOD_HLL))
        faces<true, ORDER, TX, TY, NT>(P, smem, tx0, ty0, dt_only, left, fastest);
    else
        faces<false, ORDER, TX, TY, NT>(P, smem, tx0, ty0, dt_only, left, fastest);
    __syncthreads();
    if (left.n != 0) {
        faces_left<ORDER, TX, TY, NT>(P, in, smem, tx0, ty0, left, fastest);
        __syncthreads();
    }
    update_cells<double, ORDER, TX, TY, NT, TX, TX * TY>(P, out, tx0, ty0, T_do, dt_only, t.cell, t.fx,
                                                     t.fy, res, aux);
    res.umax_x = fastest.x;
    res.umax_y = fastest.y;
}

__device__ __forceinline__ void add_counters(Scalars* ctr, const TileResult& r) {
    if (ctr != nullptr && (r.nfl_r | r.nfl_p | r.nbad)) {
        if (r.nfl_r) atomicAdd(&ctr->rho_floor, (unsigned long long)r.nfl_r);
        if (r.nfl_p) atomicAdd(&ctr->p_floor, (unsigned long long)r.nfl_p);
        if (r.nbad) atomicAdd(&ctr->nonfinite, (unsigned long long)r.nbad);
    }
}

template <int METHODS, int ORDER, int TX, int TY, int NT>
__global__ void __launch_bounds__(NT, NT == kNT ? kCtas<TX, TY> : 1) euler_fast_kernel(const __grid_constant__ Params P,
                                                        const __grid_constant__ CPlanes in,
                                                        const __grid_constant__ Planes out,
                                                        const double* __restrict__ T_do_ptr,
                                                        unsigned long long* T_bits, Scalars* rot,
                                                        Scalars* ctr, int dt_only,
                                                        double* aux) {
    extern __shared__ double smem[];
    TileResult r;
    step_tile<METHODS, ORDER, TX, TY, NT>(P, in, out, blockIdx.x * TX, (blockIdx.y + P.tile_row0) * TY,
                             *T_do_ptr, dt_only, smem, r, aux);
    add_counters(ctr, r);
    block_dt_and_rotate<NT>(P, r.umax_x, r.umax_y, r.any_active, T_bits, rot, P.tile_nblocks);
}

// Tangent of one step: (U, dU) -> dU' with the dt read from *T_do_ptr (held fixed):
// the same tile instantiated with Dual values.  32 x 8 tiles: a Dual tile holds twice the
// bytes of a double one (101 KB at second order), so two CTAs fit on an SM (at 32 x 16, 186 KB,
// one).
constexpr int kTanTX = 32, kTanTY = 8;
template <int ORDER>
__global__ void __launch_bounds__(kNTTan) euler_tangent_kernel(Params P, CPlanes in, CPlanes din,
                                                           Planes dout,
                                                           const double* __restrict__ T_do_ptr) {
    extern __shared__ __align__(16) double smem[];
    TileResult r;
    const DualIn I{in, din};
    const DualOut O{dout};
    euler_tile<Dual, ORDER, kTanTX, kTanTY, kNTTan>(P, I, O, blockIdx.x * kTanTX, blockIdx.y * kTanTY,
                                            *T_do_ptr, 0, reinterpret_cast<Dual*>(smem), r,
                                            nullptr);
}

// Persistent batched step: CTAs stride over the flattened (grid, tile) work list; each tile
// reports its dt to its own grid, and the last tile of a grid rotates that grid's dt.
// With dt_only, tiles only min-combine their dt (no state write, no rotation).
// `sc_override` (may be null) replaces every grid's scalars (the autotuner times steps
// without touching the real dt and time).
// cp.async of 4 bytes, and the wait for all of this thread's
__device__ __forceinline__ void async_copy4(void* to, const void* from) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(
                     (unsigned int)__cvta_generic_to_shared(to)), "l"(from) : "memory");
}
__device__ __forceinline__ void async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// One pass of 128 grids: 6.72 ms with 192 threads per tile (78 registers, no spills); 6.80 ms with
// 256 (64 registers: the descriptors and the prefetch on top of the step spill), 6.73 ms with
// 160.  Tiles of 512 cells, two per SM, have the registers at 256 threads.
// METHODS 1: every grid's method is HLLC (0.8 % faster than with both solvers when the cells were in
// units of the tile); 3: any.
template <int METHODS, int ORDER, int TX, int TY>
__global__ void __launch_bounds__(kNTBatch<TX, TY>, kCtas<TX, TY>) euler_batch_kernel(const BatchGrid* __restrict__ grids,
                                                         const int2* __restrict__ items,
                                                         int nitems, int cur, int dt_only,
                                                         Scalars* sc_override) {
    extern __shared__ double smem[];
    // The work items and the grids' descriptors come one tile ahead, by asynchronous copies of a
    // word a thread: read at the tile's start, the two dependent loads took 10 % of its time.
    __shared__ BatchGrid grid_of[2];
    __shared__ __align__(8) int2 item_of[2];
    constexpr int kWords = sizeof(BatchGrid) / 4;
    static_assert(sizeof(BatchGrid) % 4 == 0 && kWords <= kNTBatch<TX, TY>, "one word a thread");
    const int stride = gridDim.x;
    if (threadIdx.x < 2 && blockIdx.x + threadIdx.x * stride < nitems)
        item_of[threadIdx.x] = items[blockIdx.x + threadIdx.x * stride];
    __syncthreads();
    int2 w = item_of[0];
    if ((int)blockIdx.x < nitems && threadIdx.x < kWords)
        reinterpret_cast<unsigned int*>(&grid_of[0])[threadIdx.x] =
            reinterpret_cast<const unsigned int*>(grids + w.x)[threadIdx.x];
    int cur_slot = 0;
    for (int it = blockIdx.x; it < nitems; it += stride, cur_slot ^= 1) {
        // this tile's descriptor and the next one's item are there, the previous tile is done
        async_wait();
        __syncthreads();
        const BatchGrid& g = grid_of[cur_slot];
        const int tile = w.y;
        Scalars* sc = sc_override != nullptr ? sc_override + w.x : g.sc;
        if (it + stride < nitems) {
            w = item_of[cur_slot ^ 1];
            if (threadIdx.x < kWords)
                async_copy4(reinterpret_cast<unsigned int*>(&grid_of[cur_slot ^ 1]) + threadIdx.x,
                            reinterpret_cast<const unsigned int*>(grids + w.x) + threadIdx.x);
            if (threadIdx.x < 2 && it + 2 * stride < nitems)
                async_copy4(reinterpret_cast<int*>(&item_of[cur_slot]) + threadIdx.x,
                            reinterpret_cast<const int*>(items + it + 2 * stride) + threadIdx.x);
        }
        const long long K = g.K;
        CPlanes in{};
        Planes out{};
#pragma unroll
        for (int f = 0; f < NF; ++f) {
            in.f[f] = g.state[cur] + f * K;
            out.f[f] = g.state[cur ^ 1] + f * K;
        }
        const int tx0 = (tile % g.tiles_x) * TX, ty0 = (tile / g.tiles_x) * TY;
        const double T_do = sc->T_do;
        TileResult r;
        step_tile<METHODS, ORDER, TX, TY, kNTBatch<TX, TY>>(g.P, in, out, tx0, ty0, T_do, dt_only, smem, r, nullptr);
        add_counters(dt_only ? nullptr : sc, r);
        block_dt_and_rotate<kNTBatch<TX, TY>>(g.P, r.umax_x, r.umax_y, r.any_active, &sc->T_bits,
                                dt_only ? nullptr : sc, (unsigned int)g.ntiles);
    }
}

template <class K>
cudaError_t set_room(K* kernel, size_t bytes) {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}
template <int ORDER, int TX, int TY>
cudaError_t set_attrs() {
    constexpr size_t n = Shape<ORDER, TX, TY>::bytes;
    cudaError_t e = set_room(euler_fast_kernel<1, ORDER, TX, TY, kNT>, n);
    if (e == cudaSuccess) e = set_room(euler_fast_kernel<2, ORDER, TX, TY, kNT>, n);
    if constexpr (TX == 16 && TY == 16) {
        if (e == cudaSuccess) e = set_room(euler_fast_kernel<1, ORDER, TX, TY, kNTFew>, n);
        if (e == cudaSuccess) e = set_room(euler_fast_kernel<2, ORDER, TX, TY, kNTFew>, n);
    }
    if (e == cudaSuccess) e = set_room(euler_batch_kernel<1, ORDER, TX, TY>, n);
    if (e == cudaSuccess) e = set_room(euler_batch_kernel<3, ORDER, TX, TY>, n);
    return e;
}

template <int ORDER, int TX, int TY, int NT>
void launch_tiles(const Params& P, dim3 grid, const CPlanes& in, const Planes& out,
                  const double* T_do, unsigned long long* T_bits, Scalars* rot, Scalars* ctr,
                  int dt_only, cudaStream_t st, double* aux) {
    constexpr size_t n = Shape<ORDER, TX, TY>::bytes;
    if (P.method == GD_METHOD_HLL)
        euler_fast_kernel<2, ORDER, TX, TY, NT><<<grid, NT, n, st>>>(P, in, out, T_do, T_bits, rot,
                                                                     ctr, dt_only, aux);
    else
        euler_fast_kernel<1, ORDER, TX, TY, NT><<<grid, NT, n, st>>>(P, in, out, T_do, T_bits, rot,
                                                                     ctr, dt_only, aux);
}

template <int ORDER, int TX, int TY>
cudaError_t launch_single(const Params& P, const CPlanes& in, const Planes& out,
                          const double* T_do, unsigned long long* T_bits, Scalars* rot,
                          Scalars* ctr, int dt_only, cudaStream_t st, double* aux = nullptr) {
    const dim3 grid((P.N + TX - 1) / TX, P.tile_rows ? P.tile_rows : (P.M + TY - 1) / TY);
    if constexpr (TX == 16 && TY == 16) {
        if ((long long)grid.x * grid.y <= P.few_tiles) {
            launch_tiles<ORDER, TX, TY, kNTFew>(P, grid, in, out, T_do, T_bits, rot, ctr, dt_only,
                                                st, aux);
            return cudaGetLastError();
        }
    }
    launch_tiles<ORDER, TX, TY, kNT>(P, grid, in, out, T_do, T_bits, rot, ctr, dt_only, st, aux);
    return cudaGetLastError();
}

template <int ORDER, int TX, int TY>
cudaError_t launch_batch(const BatchGrid* grids, const int2* items, int nitems, int cur,
                         int dt_only, Scalars* sc_override, int ctas, bool hllc_only,
                         cudaStream_t st) {
    constexpr size_t n = Shape<ORDER, TX, TY>::bytes;
    if (hllc_only)
        euler_batch_kernel<1, ORDER, TX, TY><<<ctas, kNTBatch<TX, TY>, n, st>>>(grids, items, nitems, cur,
                                                                  dt_only, sc_override);
    else
        euler_batch_kernel<3, ORDER, TX, TY><<<ctas, kNTBatch<TX, TY>, n, st>>>(grids, items, nitems, cur,
                                                                  dt_only, sc_override);
    return cudaGetLastError();
}

// tile shapes of the variants: 0: 16x16 (the single-grid step's), 1: 32x8, 2: 32x16, 3: 64x8
#define GD_EULER_DISPATCH(ORDER, VAR, CALL, ARGS) \
    switch (VAR) {                                \
        case 1: return CALL<ORDER, 32, 8> ARGS;   \
        case 2: return CALL<ORDER, 32, 16> ARGS;  \
        case 3: return CALL<ORDER, 64, 8> ARGS;   \
        default: return CALL<ORDER, 16, 16> ARGS; \
    }

}  // namespace

void euler_tile_shape(int variant, int* tx, int* ty) {
    static const int shapes[kEulerVariants][2] = {{16, 16}, {32, 8}, {32, 16}, {64, 8}};
    const int v = (variant >= 0 && variant < kEulerVariants) ? variant : 0;
    *tx = shapes[v][0];
    *ty = shapes[v][1];
}

size_t euler_smem_bytes(int order, int variant) {
    switch (variant) {
        case 1: return order == 1 ? Shape<1, 32, 8>::bytes : Shape<2, 32, 8>::bytes;
        case 2: return order == 1 ? Shape<1, 32, 16>::bytes : Shape<2, 32, 16>::bytes;
        case 3: return order == 1 ? Shape<1, 64, 8>::bytes : Shape<2, 64, 8>::bytes;
        default: return order == 1 ? Shape<1, 16, 16>::bytes : Shape<2, 16, 16>::bytes;
    }
}

namespace {
template <int ORDER, int TX, int TY>
int blocks_per_sm() {
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, euler_batch_kernel<3, ORDER, TX, TY>, kNTBatch<TX, TY>,
                                                      Shape<ORDER, TX, TY>::bytes) != cudaSuccess)
        return 1;
    return n > 0 ? n : 1;
}
}  // namespace

int euler_batch_blocks_per_sm(int order, int variant) {
    if (order == 1) {
        switch (variant) {
            case 1: return blocks_per_sm<1, 32, 8>();
            case 2: return blocks_per_sm<1, 32, 16>();
            case 3: return blocks_per_sm<1, 64, 8>();
            default: return blocks_per_sm<1, 16, 16>();
        }
    }
    switch (variant) {
        case 1: return blocks_per_sm<2, 32, 8>();
        case 2: return blocks_per_sm<2, 32, 16>();
        case 3: return blocks_per_sm<2, 64, 8>();
        default: return blocks_per_sm<2, 16, 16>();
    }
}

cudaError_t prepare_euler_fast() {
    cudaError_t e = set_attrs<1, 32, 16>();
    if (e == cudaSuccess)  // Dual tiles: twice the bytes of the double ones
        e = cudaFuncSetAttribute(euler_tangent_kernel<1>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(Shape<1, kTanTX, kTanTY>::dual_bytes));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(euler_tangent_kernel<2>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(Shape<2, kTanTX, kTanTY>::dual_bytes));
    if (e == cudaSuccess) e = set_attrs<2, 32, 16>();
    if (e == cudaSuccess) e = set_attrs<1, 32, 8>();
    if (e == cudaSuccess) e = set_attrs<2, 32, 8>();
    if (e == cudaSuccess) e = set_attrs<1, 16, 16>();
    if (e == cudaSuccess) e = set_attrs<2, 16, 16>();
    if (e == cudaSuccess) e = set_attrs<1, 64, 8>();
    if (e == cudaSuccess) e = set_attrs<2, 64, 8>();
    return e;
}

cudaError_t launch_euler_fast_v(int variant, const Params& P, const CPlanes& in,
                                const Planes& out, const double* T_do,
                                unsigned long long* T_bits, Scalars* rot, Scalars* ctr,
                                int dt_only, cudaStream_t st) {
    if (P.order == 1) {
        GD_EULER_DISPATCH(1, variant, launch_single,
                          (P, in, out, T_do, T_bits, rot, ctr, dt_only, st));
    }
    GD_EULER_DISPATCH(2, variant, launch_single, (P, in, out, T_do, T_bits, rot, ctr, dt_only, st));
}

cudaError_t launch_euler_fast(const Params& P, const CPlanes& in, const Planes& out,
                              const double* T_do, unsigned long long* T_bits, Scalars* rot,
                              Scalars* ctr, int dt_only, cudaStream_t st) {
    return launch_euler_fast_v(0, P, in, out, T_do, T_bits, rot, ctr, dt_only, st);
}

cudaError_t launch_euler_tangent(const Params& P, const CPlanes& in, const CPlanes& din,
                                 const Planes& dout, const double* T_do, cudaStream_t st) {
    const dim3 grid((P.N + kTanTX - 1) / kTanTX, (P.M + kTanTY - 1) / kTanTY);
    if (P.order == 1)
        euler_tangent_kernel<1><<<grid, kNTTan, Shape<1, kTanTX, kTanTY>::dual_bytes, st>>>(
            P, in, din, dout, T_do);
    else
        euler_tangent_kernel<2><<<grid, kNTTan, Shape<2, kTanTX, kTanTY>::dual_bytes, st>>>(
            P, in, din, dout, T_do);
    return cudaGetLastError();
}

cudaError_t launch_euler_fast_aux(const Params& P, const CPlanes& in, const Planes& out,
                                  const double* T_do, unsigned long long* T_bits, Scalars* rot,
                                  Scalars* ctr, double* aux, cudaStream_t st) {
    // variant 0, the launch gd_advance makes: the recorded step is the plain step
    if (P.order == 1)
        return launch_single<1, 16, 16>(P, in, out, T_do, T_bits, rot, ctr, 0, st, aux);
    return launch_single<2, 16, 16>(P, in, out, T_do, T_bits, rot, ctr, 0, st, aux);
}

cudaError_t launch_euler_batch(int variant, int order, const BatchGrid* grids, const int2* items,
                               int nitems, int cur, int dt_only, Scalars* sc_override, int ctas,
                               bool hllc_only, cudaStream_t st) {
    if (order == 1) {
        GD_EULER_DISPATCH(1, variant, launch_batch,
                          (grids, items, nitems, cur, dt_only, sc_override, ctas, hllc_only, st));
    }
    GD_EULER_DISPATCH(2, variant, launch_batch,
                      (grids, items, nitems, cur, dt_only, sc_override, ctas, hllc_only, st));
}


namespace {
// One face per thread through the step's own face solver (hllc_local / hll_local): L, R are
// n x 4 (rho, p, vx, vy); flux n x 4 (mass, energy, x momentum, y momentum), the reference's
// HLLC_Aleksashov output order; speed n values max(|S_L|, |S_R|).  axis 0: normal +x.
__global__ void euler_face_probe_kernel(Params P, long long n, int axis,
                                        const double* __restrict__ L,
                                        const double* __restrict__ R, double* flux,
                                        double* speed) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double* a = L + 4 * i;
    const double* b = R + 4 * i;
    const bool isx = axis == 0;
    const double qa[NF] = {a[0], a[1], isx ? a[2] : a[3], isx ? a[3] : a[2]};
    const double qb[NF] = {b[0], b[1], isx ? b[2] : b[3], isx ? b[3] : b[2]};
    double UU, f[NF];
    FluxE<double> F;
    if (P.method == GD_METHOD_HLL ? fx::euler_face<true>(qa, qb, P.gas, f, UU)
                                  : fx::euler_face<false>(qa, qb, P.gas, f, UU))
        F = FluxE<double>{f[0], f[1], f[2], f[3]};
    else
        F = float_flux(P, qa, qb, UU);
    double* o = flux + 4 * i;
    o[0] = F.m;
    o[1] = F.e;
    o[2] = isx ? F.mn : F.mt;
    o[3] = isx ? F.mt : F.mn;
    speed[i] = dabs(UU);
}
}  // namespace

cudaError_t launch_euler_face_probe(const Params& P, long long n, int axis, const double* L,
                                    const double* R, double* flux, double* speed,
                                    cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    const long long blocks = (n + 255) / 256;
    euler_face_probe_kernel<<<(unsigned int)blocks, 256, 0, st>>>(P, n, axis, L, R, flux, speed);
    return cudaGetLastError();
}

}  // namespace gd
