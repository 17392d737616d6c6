// gd_fast_hancock.cu -- fast MUSCL-Hancock step (Kernel_GKR, kernel.cu:2663-3284): the
// predictor-corrector with HLLD faces, face-once on tiles, FMA contraction, field in
// Heaviside-Lorentz units (b = B / sqrt(4 pi)).
//
// The reference evaluates, for every cell, the half-step predictions of itself and of its
// four neighbours, so each prediction is computed five times and each face twice.  Away
// from the edges a cell's view of a neighbour's prediction is the neighbour's own (same
// stencil points), so here every prediction is computed once per tile and every face once.
// That holds for the cells with 2 <= n < N-2 and 2 <= m < M-2 (the "interior"); along the
// edges the reference's substitutes depend on the asking cell (see gd_hancock_cell.cuh), and
// the two-cell band is computed cell by cell exactly as the reference does.  Two launches:
//   hancock_band_kernel   the band cells, per cell (hancock_cell of gd_hancock_cell.cuh)
//   hancock_tile_kernel   32 x 8 interior tiles:
//     L  state of the tile + 2 halo (cross-shaped), B -> b
//     P  per cell of the tile + 1 halo: minmod slopes, the half step of the primitive state
//        from the differences of the predictor's physical fluxes (POTOK_Korolkov,
//        Gas_Dinamic.cu:70-180; the differences by the product rule) and sources, the
//        half-step mean A = (Q + QQ)/2
//     F  each face once: HLLD between A_L + D_L/2 and A_R - D_R/2, in scaled 64-bit integers
//        (gd_fixed_mhd.cuh), in FP64 (gd_mhd_flux.cuh) where a face's states leave their range
//     U  the corrector of kernel.cu:3256-3281 (Pdiv = 0) from A and the four faces
// Given a side stream, the band kernel runs on it concurrently with the tile kernel (they
// write disjoint cells); the blocks of both share one ticket, and the last block of either to
// finish performs the funk_time rotation.
//
// The tile kernel is bound by the FP64 pipe (71 % active): 305 FP64 operations per cell of the
// grid, most of them the predictor's; 671 with FP64 faces and a predictor in conserved
// quantities.  One step at 3226 x 1792: 4.55 ms, 8.01 ms before.
//
// Differences from the parity step are rounding only: contraction, reciprocals instead of
// divisions, slopes minmod(a - b, b - c) instead of h minmod((a - b)/h, (b - c)/h), the
// neighbour's prediction at its own radius y_{m+-1} instead of y -+ dy, and the face solved
// once (its two sides see the same flux up to rounding of the solver's symmetry).
#include "gd_fixed_mhd.cuh"
#include "gd_hancock_cell.cuh"
#include "gd_internal.cuh"
#include "gd_kernels.h"
#include "gd_mhd_flux.cuh"

namespace gd {
namespace {

constexpr int TX = 32, TY = 8, NT = TX * TY;  // one interior cell per thread in U
constexpr int NF = 7;                          // rho, p, vx, vy, bx, by, bz
constexpr int RX = TX + 4, RY = TY + 4;        // state: tile + 2
constexpr int PX = TX + 2, PY = TY + 2;        // predictions: tile + 1
constexpr int kRaw = NF * RY * RX;
constexpr int kPred = NF * PY * PX;            // one array each of A, DX, DY
constexpr int NFX = (TX + 1) * TY, NFY = TX * (TY + 1);
constexpr int kFx = NF * NFX, kFy = NF * NFY;
constexpr int kUnion = kRaw > kFx + kFy ? kRaw : kFx + kFy;  // state, later the fluxes
constexpr size_t kSmemBytes = sizeof(double) * (kUnion + 3 * kPred + 2 * PY + TX) + TX * TY;

constexpr int BNT = 128;  // band kernel

// Half the jump F(m + h) - F(m - h) of the physical flux through a face, in its local frame
// (normal velocity u, tangential v, no z velocity; field bn, bt, bz in b units), as the predictor
// (kernel.cu:1611-1720) uses it, by the product rule: for a product, (a + x)(b + y) -
// (a - x)(b - y) = 2 (a y + x b), and so on for the cubic and quartic terms.  The momenta and the
// energy come with what the predicted state takes out of them again already gone,
//   n = J(normal momentum) - u J(mass), t = J(tangential) - v J(mass),
//   i = J(energy) - u J(normal) - v J(tangential) + (u^2 + v^2)/2 J(mass) - bt J(bt) - bz J(bz),
// where all but the terms below cancel: 31 operations where the plain jumps take 45, and none of
// the update's cancellations to round.  G = gamma / (gamma - 1).
struct FluxJump {
    double m, n, t, i, bt, bz;
};
__device__ __forceinline__ FluxJump flux_jump(double r, double p, double u, double v, double bn,
                                              double bt, double bz, double rh, double ph,
                                              double uh, double vh, double bnh, double bth,
                                              double bzh, double G) {
    FluxJump J;
    const double w = fma(rh, uh, r * u);
    J.m = fma(r, uh, rh * u);
    J.n = fma(uh, w, fma(bt, bth, fma(bz, bzh, fma(-bn, bnh, ph))));
    J.t = fma(w, vh, -fma(bn, bth, bnh * bt));
    J.bt = fma(u, bth, fma(uh, bt, -fma(v, bnh, vh * bn)));
    J.bz = fma(u, bzh, uh * bz);
    const double cross = bnh * fma(u, bn, fma(v, bt, -vh * bth));
    const double mag = fma(uh, fma(bth, bth, bzh * bzh), cross);
    const double kin = fma(half_exact(J.m), fma(uh, uh, vh * vh), mag);
    J.i = fma(G, fma(p, uh, ph * u), fma(-u, ph, kin));
    return J;
}

// rho and p of the predictor's face states Q +- D/2 as mean m and half-difference h, with the
// reference's fallback to Q where a state is <= 0 (kernel.cu:1640-1680); the other fields have
// m = Q, h = D/2.
__device__ __forceinline__ void mean_half(const double* Q, const double* D, double* m,
                                          double* h) {
#pragma unroll
    for (int f = 0; f < 2; ++f) {
        // |D| < 2 Q (always, for a minmod slope between positive cells): neither state is <= 0
        if (gt_zero(Q[f]) && mag_lt(D[f], twice_exact(Q[f]))) {
            m[f] = Q[f];
            h[f] = half_exact(D[f]);
            continue;
        }
        double a = fma(0.5, D[f], Q[f]), b = fma(-0.5, D[f], Q[f]);
        a = le_zero(a) ? Q[f] : a;
        b = le_zero(b) ? Q[f] : b;
        m[f] = half_exact(a + b);
        h[f] = half_exact(a - b);
    }
}

// One face of a tile: faces 0 .. NFX-1 have an x normal, the rest a y normal.
struct FaceH {
    bool isx, used;  // used: next to a cell that the step updates
    int pa, pb, out;  // the predictions on either side, and the place among the tile's fluxes
    __device__ FaceH(const unsigned char* flag, int i) {
        isx = i < NFX;
        if (isx) {
            const int ly = i / (TX + 1), lx = i - ly * (TX + 1);
            used = (lx > 0 && flag[ly * TX + lx - 1] == 2) || (lx < TX && flag[ly * TX + lx] == 2);
            pa = (ly + 1) * PX + lx;  // cell lx-1 of the tile
            pb = pa + 1;
            out = i;
        } else {
            const int j = i - NFX, ly = j / TX, lx = j - ly * TX;
            used = (ly > 0 && flag[(ly - 1) * TX + lx] == 2) || (ly < TY && flag[ly * TX + lx] == 2);
            pa = ly * PX + lx + 1;  // cell (lx, ly-1) of the tile
            pb = pa + PX;
            out = j;
        }
    }
    // its states A + D/2 and A - D/2 in the local frame: x-face (n, t) = (x, y), y-face (y, x)
    __device__ __forceinline__ void states(const double* pA, const double* D, double* qa,
                                           double* qb) const {
#pragma unroll
        for (int f = 0; f < NF; ++f) {
            const int g = (isx || f < 2 || f == 6 ? f : (f < 4 ? 5 - f : 9 - f)) * (PY * PX);
            const double Aa = pA[g + pa], Ab = pA[g + pb];
            qa[f] = fma(0.5, D[g + pa], Aa);
            qb[f] = fma(-0.5, D[g + pb], Ab);
            if (f < 2) {
                qa[f] = le_zero(qa[f]) ? Aa : qa[f];
                qb[f] = le_zero(qb[f]) ? Ab : qb[f];
            }
        }
    }
    template <class F>
    __device__ __forceinline__ void store(double* fx, double* fy, const F& f) const {
        double* fo = (isx ? fx : fy) + out;
        const int st = isx ? NFX : NFY;
        fo[0 * st] = f.m;
        fo[1 * st] = f.e;
        fo[2 * st] = isx ? f.mn : f.mt;
        fo[3 * st] = isx ? f.mt : f.mn;
        fo[4 * st] = isx ? f.bn : f.bt;
        fo[5 * st] = isx ? f.bt : f.bn;
        fo[6 * st] = f.bz;
    }
};

// The faces that the integer solver left, in floating point.
__device__ __noinline__ void faces_left(const Params& P, double* smem, const unsigned char* flag,
                                        const LeftFaces<NFX + NFY>& left, double& umax_x,
                                        double& umax_y) {
    const double *pA = smem + kUnion, *pDX = pA + kPred, *pDY = pDX + kPred;
    for (unsigned int k = threadIdx.x; k < left.n; k += NT) {
        const FaceH w(flag, left.face(k));
        double qa[NF], qb[NF], UU;
        w.states(pA, w.isx ? pDX : pDY, qa, qb);
        Side<double> A, B;
        side(A, qa[0], qa[1], qa[2], qa[3], qa[4], qa[5], qa[6], P);
        side(B, qb[0], qb[1], qb[2], qb[3], qb[4], qb[5], qb[6], P);
        w.store(smem, smem + kFx, hlld_local(A, B, GD_METHOD_HLLD, P, UU));
        if (left.no_speed(k)) {
            if (w.isx) umax_x = max_nonneg(umax_x, UU);
            else umax_y = max_nonneg(umax_y, UU);
        }
    }
}

template <bool VYP>
__global__ void __launch_bounds__(NT, 2) hancock_tile_kernel(const __grid_constant__ Params P,
                                                          const __grid_constant__ CPlanes in,
                                                          const __grid_constant__ Planes out,
                                                          const double* __restrict__ T_do_ptr,
                                                          unsigned long long* T_bits,
                                                          Scalars* rot, Scalars* ctr,
                                                          int dt_only, unsigned int nblocks) {
    extern __shared__ __align__(16) double smem[];
    double* raw = smem;            // [NF][RY][RX], then fx [NF][TY][TX+1], fy [NF][TY+1][TX]
    double* fx = smem;
    double* fy = smem + kFx;
    double* pA = smem + kUnion;    // [NF][PY][PX]
    double* pDX = pA + kPred;
    double* pDY = pDX + kPred;
    double* rowy = pDY + kPred;    // radius of prediction rows
    double* rowiy = rowy + PY;     // its reciprocal
    double* colx = rowiy + PY;     // x of the tile's columns
    unsigned char* flag = reinterpret_cast<unsigned char*>(colx + TX);  // [TY][TX]
    __shared__ LeftFaces<NFX + NFY> left;

    const int tid = threadIdx.x;
    if (tid == 0) left.n = 0;
    const int N = P.N, M = P.M;
    const int tx0 = 2 + blockIdx.x * TX, ty0 = 2 + (blockIdx.y + P.tile_row0) * TY;

    // ---- L: state of the tile + 2 halo; corner blocks the stencils never reach are skipped
    for (int i = tid; i < RY * RX; i += NT) {
        const int ly = i / RX, lx = i - ly * RX;
        if ((lx == 0 || lx == RX - 1) && (ly < 2 || ly >= TY + 2)) continue;
        if ((ly == 0 || ly == RY - 1) && (lx < 2 || lx >= TX + 2)) continue;
        const int gx = tx0 + lx - 2, gy = ty0 + ly - 2;
        double v[NF];
        if (gx >= 0 && gx < N && gy >= 0 && gy < M) {
            const long long k = (long long)gy * N + gx;
#pragma unroll
            for (int f = 0; f < NF; ++f) v[f] = load_f(in, f, k);
            v[4] *= kInvSpi4;
            v[5] *= kInvSpi4;
            v[6] *= kInvSpi4;
        } else {
            // outside the grid: only predictions that no interior face uses read these
#pragma unroll
            for (int f = 0; f < NF; ++f) v[f] = f < 2 ? 1.0 : 0.0;
        }
#pragma unroll
        for (int f = 0; f < NF; ++f) raw[(f * RY + ly) * RX + lx] = v[f];
    }
    if (tid < PY) {
        const double y = hancock_y(P, ty0 + tid - 1);
        rowy[tid] = y;
        rowiy[tid] = 1.0 / y;
    } else if (tid >= 32 && tid < 32 + TX) {
        colx[tid - 32] = hancock_x(P, tx0 + tid - 32);
    }
    __syncthreads();
    // this thread's cell: 0 outside the interior, 1 interior and frozen, 2 interior, updated
    const int cx = tid % TX, cy = tid / TX;
    const int gx = tx0 + cx, gy = ty0 + cy;
    int my_flag = 0;
    if (gx < N - 2 && gy < M - 2) my_flag = hancock_frozen_fast(P, colx[cx], rowy[cy + 1]) ? 1 : 2;
    flag[tid] = (unsigned char)my_flag;
    // a tile inside the frozen sphere has nothing to predict or solve (7 % of the wind's tiles)
    const bool any_active = __syncthreads_or(my_flag == 2) != 0;
    if (!any_active) {
        if (my_flag == 1 && !dt_only) {
            const long long k = (long long)gy * N + gx;
#pragma unroll
            for (int f = 0; f < NF; ++f) store_f(out, f, k, load_f(in, f, k));
        }
        block_dt_and_rotate<NT>(P, 0.0, 0.0, false, T_bits, rot, nblocks);
        return;
    }

    // ---- P: predictions of the tile + 1 halo (not its corners) ---------------------------
    const double T_do = *T_do_ptr;
    const double st = 0.5 * T_do;
    const double sx = st * P.inv_dx, sy = st * P.inv_dy;
    const double sx2 = twice_exact(sx), sy2 = twice_exact(sy);
    for (int i = tid; i < PY * PX; i += NT) {
        const int py = i / PX, px = i - py * PX;
        if ((px == 0 || px == PX - 1) && (py == 0 || py == PY - 1)) continue;
        const double* c = raw + (py + 1) * RX + (px + 1);
        constexpr int PS = RY * RX;
        double Q[NF], DX[NF], DY[NF];
#pragma unroll
        for (int f = 0; f < NF; ++f) {
            const double* q = c + f * PS;
            Q[f] = q[0];
            DX[f] = minmod(q[1] - q[0], q[0] - q[-1]);
            DY[f] = minmod(q[RX] - q[0], q[0] - q[-RX]);
        }
        if (VYP) {
            DX[3] = DX[1];
            DY[3] = DY[1];
        }
        // predictor (kernel.cu:1611-1720) with the flux differences of the face states Q +- D/2,
        // 2 sx J_x + 2 sy J_y (x: normal u, field bx; y: normal v, by) and the sources of y, as
        // changes of the primitive state:
        //   rho' = rho - dr, u' = u - Mu / rho', v' = v - Mv / rho', b' = b - db,
        //   p' = p - (gamma - 1) (W + (Mu^2 + Mv^2) / (2 rho') + |db|^2 / 2)
        double mx[2], hx[2], my[2], hy[2];  // rho and p
        mean_half(Q, DX, mx, hx);
        mean_half(Q, DY, my, hy);
        const double r = Q[0], p = Q[1], u = Q[2], v = Q[3], bx = Q[4], by = Q[5], bz = Q[6];
        const FluxJump Jx = flux_jump(mx[0], mx[1], u, v, bx, by, bz, hx[0], hx[1],
                                      half_exact(DX[2]), half_exact(DX[3]), half_exact(DX[4]),
                                      half_exact(DX[5]), half_exact(DX[6]), P.g_gm1);
        const FluxJump Jy = flux_jump(my[0], my[1], v, u, by, bx, bz, hy[0], hy[1],
                                      half_exact(DY[3]), half_exact(DY[2]), half_exact(DY[5]),
                                      half_exact(DY[4]), half_exact(DY[6]), P.g_gm1);
        const double sty = st * rowiy[py];
        const double dr = fma(sty * r, v, fma(sy2, Jy.m, sx2 * Jx.m));
        const double Mu = fma(sy2, Jy.t, fma(sx2, Jx.n, -sty * (bx * by)));
        const double Mv = fma(sy2, Jy.n, fma(sx2, Jx.t, sty * fma(bz, bz, -by * by)));
        const double dbx = fma(sy2, Jy.bt, sty * fma(v, bx, -by * u));
        const double dby = sx2 * Jx.bt;
        const double dbz = fma(sy2, Jy.bz, sx2 * Jx.bz);
        const double ub = fma(u, bx, v * by);
        const double W = fma(sx2, Jx.i, fma(sy2, Jy.i, sty * fma(p * P.g_gm1, v, by * ub)));
        const double db2 = fma(dbz, dbz, fma(dby, dby, dbx * dbx));
        const double r2 = r - dr;
        double Ar, Ap, Au, Av;  // (Q + Q') / 2
        if (le_zero(r2)) {  // rho' <= 0 keeps rho (kernel.cu:1690): from the conserved values
            const double u2 = fma(u, r2, -Mu) / r, v2 = fma(v, r2, -Mv) / r;
            const double b0 = bx - dbx, b1 = by - dby, b2 = bz - dbz;
            const double E2 = fma(p, P.inv_gm1, 0.5 * fma(r2, fma(u, u, v * v),
                                                          fma(bz, bz, fma(by, by, bx * bx)))) -
                              W - fma(u, Mu, v * Mv) - fma(bx, dbx, fma(by, dby, bz * dbz));
            double p2 = (E2 - 0.5 * fma(r, fma(u2, u2, v2 * v2),
                                        fma(b0, b0, fma(b1, b1, b2 * b2)))) * P.gm1;
            p2 = le_zero(p2) ? 0.000001 : p2;
            Ar = r;
            Ap = half_exact(p + p2);
            Au = half_exact(u + u2);
            Av = half_exact(v + v2);
        } else {
            const double ir2 = rcp_fast(r2);
            const double du = Mu * ir2, dv = Mv * ir2;
            const double dp = P.gm1 * fma(0.5, fma(Mu, du, fma(Mv, dv, db2)), W);
            const double p2 = p - dp;
            Ar = fma(-0.5, dr, r);
            Ap = le_zero(p2) ? half_exact(p + 0.000001) : fma(-0.5, dp, p);
            Au = fma(-0.5, du, u);
            Av = fma(-0.5, dv, v);
        }
        const double A[NF] = {Ar, Ap, Au, Av, fma(-0.5, dbx, bx), fma(-0.5, dby, by),
                              fma(-0.5, dbz, bz)};
        const int o = py * PX + px;
#pragma unroll
        for (int f = 0; f < NF; ++f) {
            pA[f * PY * PX + o] = A[f];
            pDX[f * PY * PX + o] = DX[f];
            pDY[f * PY * PX + o] = DY[f];
        }
    }
    __syncthreads();

    // ---- F: each face of an updated cell once: HLLD in 64-bit integers (gd_fixed_mhd.cuh), the
    // two states of a face in units of their own; the corrector and the predictor keep the FP64
    // pipe (the flux took 240 of the step's 671 FP64 operations a cell)
    double umax_x = 0.0, umax_y = 0.0;
    for (int i = tid; i < NFX + NFY; i += NT) {
        const FaceH w(flag, i);
        if (!w.used) continue;
        double qa[NF], qb[NF], UU;
        w.states(pA, w.isx ? pDX : pDY, qa, qb);
        fx::i64 a[NF], b[NF];
        int top[NF];
        fx::FluxI F;
        bool speed_ok = false, done = false;
        if (fx::face_units(qa, qb, P.gas, a, b, top))
            done = fx::mhd_face_flux<true>(a, b, top, P.gas, F, UU, speed_ok, dt_only);
        if (speed_ok) {
            if (w.isx) umax_x = max_nonneg(umax_x, UU);
            else umax_y = max_nonneg(umax_y, UU);
        }
        if (!done) left.add(i, speed_ok);
        else if (!dt_only) w.store(fx, fy, F);
    }
    __syncthreads();
    if (left.n != 0) {
        faces_left(P, smem, flag, left, umax_x, umax_y);
        __syncthreads();
    }

    // ---- U: corrector (kernel.cu:3256-3281, Pdiv = 0) --------------------------------------
    unsigned int nfl_r = 0, nfl_p = 0, nbad = 0;
    if (my_flag == 1 && !dt_only) {
        const long long k = (long long)gy * N + gx;
#pragma unroll
        for (int f = 0; f < NF; ++f) store_f(out, f, k, load_f(in, f, k));
    } else if (my_flag == 2 && !dt_only) {
        const double hT = 0.5 * T_do;
        const double kx = hT * P.inv_dx, ky = hT * P.inv_dy;
        const double hTy = hT * rowiy[cy + 1];
        const int o = (cy + 1) * PX + (cx + 1);
        double A[NF], d[NF];
#pragma unroll
        for (int f = 0; f < NF; ++f) {
            A[f] = pA[f * PY * PX + o];
            const double* a = fx + f * NFX + cy * (TX + 1) + cx;
            const double* b = fy + f * NFY + cy * TX + cx;
            d[f] = fma(kx, a[1] - a[0], ky * (b[TX] - b[0]));
        }
        const double r = A[0], p = A[1], u = A[2], v = A[3], bx = A[4], by = A[5], bz = A[6];
        const double bb = fma(bz, bz, fma(by, by, bx * bx));
        const double K1 = fma(r, fma(u, u, v * v), bb);
        double r2 = fma(-hTy * r, v, r - d[0]);
        if (le_zero(r2)) {
            r2 = r;
            ++nfl_r;
        }
        const double ir2 = rcp_fast(r2);
        const double u2 = fma(-hTy, fma(r * u, v, -bx * by), fma(r, u, -d[2])) * ir2;
        const double v2 = fma(-hTy, fma(r * v, v, fma(bz, bz, -by * by)), fma(r, v, -d[3])) * ir2;
        const double bx2 = fma(-hTy, fma(v, bx, -by * u), bx - d[4]);
        const double by2 = by - d[5];
        const double bz2 = bz - d[6];
        const double dE = fma(hTy, fma(fma(p, P.g_gm1, half_exact(K1 + bb)), v,
                                       -by * fma(u, bx, v * by)), d[1]);
        const double K2 = fma(r2, fma(u2, u2, v2 * v2), fma(bz2, bz2, fma(by2, by2, bx2 * bx2)));
        double p2 = fma(P.hgm1, K1 - K2, fma(-P.gm1, dE, p));
        if (le_zero(p2)) {
            p2 = 0.000001;
            ++nfl_p;
        }
        if (!finite_bits(r2) || !finite_bits(p2) || !finite_bits(u2) || !finite_bits(v2) ||
            !finite_bits(bx2) || !finite_bits(by2) || !finite_bits(bz2))
            ++nbad;
        const long long k = (long long)gy * N + gx;
        store_f(out, 0, k, r2);
        store_f(out, 1, k, p2);
        store_f(out, 2, k, u2);
        store_f(out, 3, k, v2);
        store_f(out, 4, k, bx2 * kSpi4);
        store_f(out, 5, k, by2 * kSpi4);
        store_f(out, 6, k, bz2 * kSpi4);
    }
    if (ctr != nullptr && (nfl_r | nfl_p | nbad)) {
        if (nfl_r) atomicAdd(&ctr->rho_floor, (unsigned long long)nfl_r);
        if (nfl_p) atomicAdd(&ctr->p_floor, (unsigned long long)nfl_p);
        if (nbad) atomicAdd(&ctr->nonfinite, (unsigned long long)nbad);
    }
    block_dt_and_rotate<NT>(P, umax_x, umax_y, any_active, T_bits, rot, nblocks);
}

// The edge cells of rows [r0, r1): rows m < 2 and m >= M-2 whole, and the columns n < 2 and
// n >= N-2 of the rows between.
struct Band {
    int lo0, nlo;    // whole rows [lo0, lo0 + nlo) at the bottom
    int hi0, nhi;    // whole rows [hi0, hi0 + nhi) at the top
    int mid0, nmid;  // rows [mid0, mid0 + nmid) between, their edge columns only
    int cols_lo, cols_hi0, ncols;
    int total;
};

int clamp_count(int a, int b) { return b > a ? b - a : 0; }

Band make_band(int N, int M, int r0, int r1) {
    Band b;
    const int bot = M < 2 ? M : 2;           // rows [0, bot) are whole
    const int top = M - 2 > 2 ? M - 2 : 2;   // rows [top, M) are whole
    b.lo0 = r0;
    b.nlo = clamp_count(r0, r1 < bot ? r1 : bot);
    b.hi0 = r0 > top ? r0 : top;
    b.nhi = clamp_count(b.hi0, r1 < M ? r1 : M);
    b.mid0 = r0 > bot ? r0 : bot;
    b.nmid = clamp_count(b.mid0, r1 < top ? r1 : top);
    b.cols_lo = N < 2 ? N : 2;
    b.cols_hi0 = N - 2 > 2 ? N - 2 : 2;
    b.ncols = b.cols_lo + (N - b.cols_hi0);
    b.total = (b.nlo + b.nhi) * N + b.nmid * b.ncols;
    return b;
}

template <bool VYP>
__global__ void __launch_bounds__(BNT) hancock_band_kernel(Params P, CPlanes in, Planes out,
                                                           const double* __restrict__ T_do_ptr,
                                                           unsigned long long* T_bits,
                                                           Scalars* rot, Scalars* ctr,
                                                           int dt_only, Band b,
                                                           unsigned int nblocks) {
    const int i = blockIdx.x * BNT + threadIdx.x;
    double tmin = kCellTmin0;
    bool active = false;
    unsigned int nfl_r = 0, nfl_p = 0, nbad = 0;
    if (i < b.total) {
        int n, m;
        if (i < (b.nlo + b.nhi) * P.N) {
            const int r = i / P.N;
            n = i - r * P.N;
            m = r < b.nlo ? b.lo0 + r : b.hi0 + (r - b.nlo);
        } else {
            const int j = i - (b.nlo + b.nhi) * P.N;
            const int r = j / b.ncols, c = j - r * b.ncols;
            m = b.mid0 + r;
            n = c < b.cols_lo ? c : b.cols_hi0 + (c - b.cols_lo);
        }
        const long long k = (long long)m * P.N + n;
        const double y = hancock_y(P, m);
        if (hancock_frozen(P, n, y)) {
            if (!dt_only)
                for (int f = 0; f < NF; ++f) store_f(out, f, k, load_f(in, f, k));
        } else {
            active = true;
            double res[NF];
            tmin = hancock_cell<VYP>(P, in, n, m, y, *T_do_ptr, res, nfl_r, nfl_p);
            if (!dt_only) {
                for (int f = 0; f < NF; ++f) {
                    if (!finite_bits(res[f])) {
                        ++nbad;
                        break;
                    }
                }
                for (int f = 0; f < NF; ++f) store_f(out, f, k, res[f]);
            }
        }
    }
    if (ctr != nullptr && !dt_only && (nfl_r | nfl_p | nbad)) {
        if (nfl_r) atomicAdd(&ctr->rho_floor, (unsigned long long)nfl_r);
        if (nfl_p) atomicAdd(&ctr->p_floor, (unsigned long long)nfl_p);
        if (nbad) atomicAdd(&ctr->nonfinite, (unsigned long long)nbad);
    }
    block_tmin_and_rotate<BNT>(tmin, active, T_bits, rot, nblocks);
}

// Interior tile rows (at least one launch row, so a step always has a tile block) and the
// tile rows [t0, t1) of the rows [r0, r1), whose ends are 0, M or 2 + a multiple of TY.
int tile_rows_all(const Params& P) { return P.M - 4 > 0 ? (P.M - 4 + TY - 1) / TY : 1; }
void tile_range(const Params& P, int r0, int r1, int* t0, int* t1) {
    *t0 = r0 <= 2 ? 0 : (r0 - 2) / TY;
    *t1 = r1 >= P.M ? tile_rows_all(P) : (r1 - 2) / TY;
}
int tile_cols(const Params& P) { return P.N - 4 > 0 ? (P.N - 4 + TX - 1) / TX : 1; }

template <bool VYP>
cudaError_t launch_rows(const Params& P0, const CPlanes& in, const Planes& out,
                        const double* T_do, unsigned long long* T_bits, Scalars* rot,
                        Scalars* ctr, int r0, int r1, unsigned int nblocks, int parts,
                        cudaStream_t st) {
    const Band b = make_band(P0.N, P0.M, r0, r1);
    int t0, t1;
    tile_range(P0, r0, r1, &t0, &t1);
    Params P = P0;
    P.tile_row0 = t0;
    if ((parts & 1) && b.total > 0)
        hancock_band_kernel<VYP><<<(b.total + BNT - 1) / BNT, BNT, 0, st>>>(
            P, in, out, T_do, T_bits, rot, ctr, 0, b, nblocks);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess || !(parts & 2) || t1 <= t0) return e;
    hancock_tile_kernel<VYP><<<dim3(tile_cols(P), t1 - t0), NT, kSmemBytes, st>>>(
        P, in, out, T_do, T_bits, rot, ctr, 0, nblocks);
    return cudaGetLastError();
}

template <bool VYP>
cudaError_t launch_v(const Params& P, const CPlanes& in, const Planes& out, const double* T_do,
                     unsigned long long* T_bits, Scalars* rot, Scalars* ctr, int dt_only,
                     cudaStream_t st, const HancockStreams* side) {
    const Band b = make_band(P.N, P.M, 0, P.M);
    const unsigned int band_blocks = (b.total + BNT - 1) / BNT;
    const int nx = tile_cols(P), ny = tile_rows_all(P);
    const unsigned int total = band_blocks + (unsigned int)(nx * ny);
    cudaStream_t bs = st;
    cudaError_t e;
    if (side != nullptr) {
        e = cudaEventRecord(side->fork, st);
        if (e == cudaSuccess) e = cudaStreamWaitEvent(side->stream, side->fork, 0);
        if (e != cudaSuccess) return e;
        bs = side->stream;
    }
    hancock_band_kernel<VYP><<<band_blocks, BNT, 0, bs>>>(P, in, out, T_do, T_bits, rot, ctr,
                                                          dt_only, b, total);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    hancock_tile_kernel<VYP><<<dim3(nx, ny), NT, kSmemBytes, st>>>(P, in, out, T_do, T_bits, rot,
                                                                   ctr, dt_only, total);
    e = cudaGetLastError();
    if (e != cudaSuccess || side == nullptr) return e;
    e = cudaEventRecord(side->join, side->stream);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(st, side->join, 0);
    return e;
}

}  // namespace

cudaError_t prepare_hancock_fast() {
    cudaError_t e = cudaFuncSetAttribute(hancock_tile_kernel<true>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)kSmemBytes);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(hancock_tile_kernel<false>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBytes);
    return e;
}

int hancock_tile_height() { return TY; }

unsigned int hancock_fast_blocks(const Params& P, int r0, int r1, int parts) {
    const Band b = make_band(P.N, P.M, r0, r1);
    int t0, t1;
    tile_range(P, r0, r1, &t0, &t1);
    return ((parts & 1) ? (unsigned int)((b.total + BNT - 1) / BNT) : 0u) +
           ((parts & 2) && t1 > t0 ? (unsigned int)((t1 - t0) * tile_cols(P)) : 0u);
}

cudaError_t launch_hancock_fast_rows(const Params& P, const CPlanes& in, const Planes& out,
                                     const double* T_do, unsigned long long* T_bits,
                                     Scalars* rot, Scalars* ctr, int r0, int r1,
                                     unsigned int nblocks, int parts, cudaStream_t st) {
    if (P.scheme == GD_SCHEME_HANCOCK_REF)
        return launch_rows<true>(P, in, out, T_do, T_bits, rot, ctr, r0, r1, nblocks, parts,
                                 st);
    return launch_rows<false>(P, in, out, T_do, T_bits, rot, ctr, r0, r1, nblocks, parts, st);
}

cudaError_t launch_hancock_fast(const Params& P, const CPlanes& in, const Planes& out,
                                const double* T_do, unsigned long long* T_bits, Scalars* rot,
                                Scalars* ctr, int dt_only, cudaStream_t st,
                                const HancockStreams* side) {
    if (P.scheme == GD_SCHEME_HANCOCK_REF)
        return launch_v<true>(P, in, out, T_do, T_bits, rot, ctr, dt_only, st, side);
    return launch_v<false>(P, in, out, T_do, T_bits, rot, ctr, dt_only, st, side);
}

}  // namespace gd
