// Point and tile functions of the split-explicit 2D substep, shared by the
// one-operation kernels (split2d.cu, momentum.cu, grid_ops.cu) and the substep's
// kernels (substep2d.cu: one domain's four, its phases, many domains' batch), so
// that every operation has a single definition and all give the same results
// bit for bit.
//
// Layout: every field is [j][i] with the full halo-inclusive extents of its
// grid (nx_, ny_ for T, U, V and their velocity grids, nx_+1, ny_+1 for X).
#pragma once

#include <math.h>

#include <type_traits>

#include "getm_common.cuh"


// torch.clamp(x, min=lo) (NaN propagates), minima and maxima with the
// comparisons on the integer pipe (the same values; an FP64 comparison costs
// as much as a multiplication)
__device__ __forceinline__ double dclamp_min(double x, double lo)
{
    return getm_isnan_i(x) ? x : (getm_dkey(x) < getm_dkey(lo) ? lo : x);
}

struct DepthArgs {
    int nx, ny;                 // T-grid extents (halos included)
    double Dmin, Dcrit, ialpha; // ialpha = 1 / (Dcrit - 2 Dmin)
    const double *z, *zo;       // elevations (T)
    const double *HT, *HU, *HV, *HX;
    const int *mT, *mU, *mV, *mX;
    double *DT, *DclipT, *workT;
    double *workU, *DU, *alphaU;
    double *workV, *DV, *alphaV;
    double *workX, *DX;         // X extents (nx+1) x (ny+1)
    double *DUU, *DVV, *DUV, *DVU;
};

constexpr int UD_BX = 32;  // tile width of update_depth_2d_tile

// alpha (wrapper.F90:428-436) with the constant divisor as a reciprocal
__device__ __forceinline__ double alpha_of(double d, double twoDmin, double ialpha)
{
    return getm_fmax_i(0.0, getm_fmin_i(1.0, (d - twoDmin) * ialpha));
}

// ... in float, for the mixed form: alpha is a weight between 0 and 1 that
// the mixed transport update reads as a float
__device__ __forceinline__ double alpha_of_f(double d, float twoDmin, float ialpha)
{
    return getm_f2d(fmaxf(0.f, fminf(1.f, (getm_d2f_approx(d) - twoDmin) * ialpha)));
}

// Simulation.update_depth, 2D part (simulation.py:1498-1586 without the
// halo exchanges and mirroring of a single closed domain).  A 32 x BY block
// covers X points (j, i) of its tile and the T, U, V points with the same
// indices; z_T_half of the tile plus a one-point halo is formed once into
// shared memory.  Copies between grids are scattered by the point that
// owns the source value (UU.D(j, i-1) = D_T_half(j, i), VV.D(j-1, i) =
// D_T_half(j, i), UV.D(j-1, i-1) = VU.D(j-1, i-1) = X.D(j, i)).
// MIXED: alpha in float (alpha_of_f); the sums stay FP64.
template <int BY, bool MIXED = false>
__device__ __forceinline__ void update_depth_2d_tile(const DepthArgs& a, int bx, int by, int tx, int ty,
                                                     double (&szh)[BY + 2][UD_BX + 2])
{
    // szh: z_T_half at rows j0-1.., cols i0-1..
    const int i0 = bx * UD_BX, j0 = by * BY;
    const int i = i0 + tx, j = j0 + ty;
    const int nx = a.nx, ny = a.ny;
    // the point's own operands, loaded while the tile is staged
    const bool xin = i <= nx && j <= ny, tin = i < nx && j < ny;
    const long long px = (long long)j * (nx + 1) + i;
    const long long p = (long long)j * nx + i;
    int mX = 0, mT = 0, mU = 0, mV = 0;
    double workX0 = 0.0, DX0 = 0.0, HX = 0.0, DT0 = 0.0, HT = 0.0, zT = 0.0, workU0 = 0.0, HU = 0.0;
    double workV0 = 0.0, HV = 0.0;
    if (xin) {
        mX = a.mX[px]; workX0 = a.workX[px]; DX0 = a.DX[px]; HX = a.HX[px];
    }
    if (tin) {
        mT = a.mT[p]; DT0 = a.DT[p]; HT = a.HT[p]; zT = a.z[p];
        mU = a.mU[p]; workU0 = a.workU[p]; HU = a.HU[p];
        mV = a.mV[p]; workV0 = a.workV[p]; HV = a.HV[p];
    }
    for (int q = ty * UD_BX + tx; q < (BY + 2) * (UD_BX + 2); q += UD_BX * BY) {
        const int sj = q / (UD_BX + 2), si = q - sj * (UD_BX + 2);
        const int gj = j0 - 1 + sj, gi = i0 - 1 + si;
        double v = 0.0;
        if (gj >= 0 && gj < ny && gi >= 0 && gi < nx) {
            const long long g = (long long)gj * nx + gi;
            v = getm_half(a.zo[g] + a.z[g]);
        }
        szh[sj][si] = v;
    }
    __syncthreads();
    if (!xin) return;
    const int sj = ty + 1, si = tx + 1;  // (j, i) in the tile
    // X point (j, i): interp_xy T->X (offsets 1, 1) where it writes, else the
    // previous X._work value
    {
        double zx;
        if (j >= 1 && j <= ny - 1 && i >= 1 && i <= nx - 1) {
            zx = getm_quarter(szh[sj - 1][si - 1] + szh[sj - 1][si] + szh[sj][si - 1] + szh[sj][si]);
            a.workX[px] = zx;
        } else {
            zx = workX0;
        }
        double dx = DX0;
        if (mX != 0) {
            dx = getm_fmax_i(HX + zx, a.Dmin);
            a.DX[px] = dx;
        }
        if (j >= 1 && i >= 1 && j - 1 < ny && i - 1 < nx) {  // UV.D = X.D[1:, 1:]; VU.D = UV.D
            const long long q = (long long)(j - 1) * nx + (i - 1);
            a.DUV[q] = dx;
            a.DVU[q] = dx;
        }
    }
    if (!tin) return;
    const double zh = szh[sj][si];
    // T: elevation2depth(z, H, -1000), Dclip = clamp(D, Dmin), D_T_half
    double DT = DT0;
    if (mT != 0) DT = getm_fmax_i(HT + zT, -1000.0);
    a.DT[p] = DT;
    a.DclipT[p] = dclamp_min(DT, a.Dmin);
    const double dth = mT != 0 ? getm_fmax_i(HT + zh, a.Dmin) : zh;
    a.workT[p] = dth;
    if (i >= 1) a.DUU[p - 1] = dth;   // UU.D[:, :-1] = D_T_half[:, 1:]
    if (j >= 1) a.DVV[p - nx] = dth;  // VV.D[:-1, :] = D_T_half[1:, :]
    const double twoDmin = 2 * a.Dmin;
    const float twoDmin_f = 2.f * getm_d2f_approx(a.Dmin), ialpha_f = getm_d2f_approx(a.ialpha);
    // U: z_U = interp_x(z_T_half, ioffset 0) for i < nx-1, else the old value
    double zu;
    if (i < nx - 1) {
        zu = getm_half(zh + szh[sj][si + 1]);
        a.workU[p] = zu;
    } else {
        zu = workU0;
    }
    if (mU != 0) {
        const double d = getm_fmax_i(HU + zu, a.Dmin);
        a.DU[p] = d;
        a.alphaU[p] = MIXED ? alpha_of_f(d, twoDmin_f, ialpha_f) : alpha_of(d, twoDmin, a.ialpha);
    }
    // V: z_V = interp_y(z_T_half, joffset 0) for j < ny-1
    double zv;
    if (j < ny - 1) {
        zv = getm_half(zh + szh[sj + 1][si]);
        a.workV[p] = zv;
    } else {
        zv = workV0;
    }
    if (mV != 0) {
        const double d = getm_fmax_i(HV + zv, a.Dmin);
        a.DV[p] = d;
        a.alphaV[p] = MIXED ? alpha_of_f(d, twoDmin_f, ialpha_f) : alpha_of(d, twoDmin, a.ialpha);
    }
}

// Momentum._transport_2d_momentum up to the advection calls
// (momentum.py:1017-1040 with Am = 0): u1 = U/DU, v1 = V/DV, the advected
// copies, and the advection velocities on the UU, UV, VU, VV grids.
// C: arithmetic of the four advection velocities (float in the mixed form).
struct VelArgs {
    int nx, ny;
    const double *U, *V, *DU, *DV, *DUU, *DUV, *DVU, *DVV;
    double *u1, *v1, *advU, *advV, *uua, *uva, *vua, *vva;
};

template <typename C>
__device__ __forceinline__ double vel_div(double num, double den)
{
    if constexpr (std::is_same<C, double>::value) return getm_div(num, den);
    else return getm_f2d(getm_d2f_approx(num) / getm_d2f_approx(den));
}

// Mixed form: u1 = U/D to ~2^-46 (getm_div_refined; u1 is advected and its
// product with the new depth is differenced against U, so it stays FP64) and
// the advection velocities entirely in float.
// One direction's: its transport T at the point and its neighbours (east at
// i + 1, north at j + 1, where they exist) over the depth D of its grid and
// those of the two advection velocity grids, De and Dn.
template <typename C>
__device__ __forceinline__ void momentum_2d_velocities_half(const VelArgs& a, int d, long long p, bool east, bool north,
                                                            double T, double Te, double Tn, double D, double De,
                                                            double Dn)
{
    double *vel = d == 0 ? a.u1 : a.v1, *adv = d == 0 ? a.advU : a.advV;
    double *ve = d == 0 ? a.uua : a.uva, *vn = d == 0 ? a.vua : a.vva;
    // interp_x (ioffset 0) writes i < nx-1; elsewhere the old value is divided
    if constexpr (std::is_same<C, double>::value) {
        const double v = getm_div(T, D);
        vel[p] = v; adv[p] = v;
        ve[p] = vel_div<C>(east ? getm_half(T + Te) : ve[p], De);
        vn[p] = vel_div<C>(north ? getm_half(T + Tn) : vn[p], Dn);
    } else {
        const double v = getm_div_refined(T, D);
        vel[p] = v; adv[p] = v;
        const float Tf = getm_d2f_approx(T);
        const float te = east ? 0.5f * (Tf + getm_d2f_approx(Te)) : getm_d2f_approx(ve[p]);
        const float tn = north ? 0.5f * (Tf + getm_d2f_approx(Tn)) : getm_d2f_approx(vn[p]);
        ve[p] = getm_f2d(te / getm_d2f_approx(De));
        vn[p] = getm_f2d(tn / getm_d2f_approx(Dn));
    }
}

template <typename C>
__device__ __forceinline__ void momentum_2d_velocities_point(const VelArgs& a, int i, int j)
{
    const long long p = (long long)j * a.nx + i;
    const bool east = i < a.nx - 1, north = j < a.ny - 1;
    momentum_2d_velocities_half<C>(a, 0, p, east, north, a.U[p], east ? a.U[p + 1] : 0.0, north ? a.U[p + a.nx] : 0.0,
                                   a.DU[p], a.DUU[p], a.DVU[p]);
    momentum_2d_velocities_half<C>(a, 1, p, east, north, a.V[p], east ? a.V[p + 1] : 0.0, north ? a.V[p + a.nx] : 0.0,
                                   a.DV[p], a.DUV[p], a.DVV[p]);
}

// Momentum.bottom_friction (momentum.py:1099-1125): u1 -> V grid and v1 -> U
// grid by interp_xy, then bottom_friction on both grids (momentum.F90:79-101,
// iterate = 0).  C: arithmetic of the drag coefficient.
struct FricArgs {
    int nx, ny;
    const int *mU, *mV;
    const double *u1, *v1, *DU, *DV, *z0bU, *z0bV;
    double *workU, *workV, *ru, *rv;
};

template <typename C>
__device__ __forceinline__ C to_c(double x)
{
    if constexpr (std::is_same<C, double>::value) return x;
    else return getm_d2f_approx(x);
}

template <typename C>
__device__ __forceinline__ double from_c(C x)
{
    if constexpr (std::is_same<C, double>::value) return x;
    else return getm_f2d(x);
}

template <typename C>
__device__ __forceinline__ C quotient(C n, C d)
{
    if constexpr (std::is_same<C, double>::value) return getm_div(n, d);
    else return n / d;
}

template <typename C>
__device__ __forceinline__ double drag(C uu, C vv, double D, double z0)
{
    const C x = C(0.5) * to_c<C>(D);
    const C sqrtcd = quotient(C(GETM_KAPPA), log(C(1) + quotient(x, to_c<C>(z0))));
    return from_c<C>(sqrtcd * sqrtcd * sqrt(getm_speed2(uu, vv)));
}

// of the U equation (d 0) or the V equation (d 1)
template <typename C>
__device__ __forceinline__ void momentum_2d_friction_half(const FricArgs& a, int d, int i, int j)
{
    const int nx = a.nx, p = j * nx + i;
    const bool u = d == 0;
    // the point's own operands, loaded before any mask is tested
    const int m = (u ? a.mU : a.mV)[p];
    const double own = (u ? a.u1 : a.v1)[p], D = (u ? a.DU : a.DV)[p], z0 = (u ? a.z0bU : a.z0bV)[p];
    const double* __restrict__ src = u ? a.v1 : a.u1;
    double* work = u ? a.workU : a.workV;
    // v_U = interp_xy(v1, ioffset 0, joffset 1): written at j >= 1, i <= nx-2;
    // u_V = interp_xy(u1, ioffset 1, joffset 0): written at i >= 1, j <= ny-2
    // (in arithmetic C: the drag coefficient is evaluated in C)
    C other;
    if (u ? j >= 1 && i <= nx - 2 : i >= 1 && j <= a.ny - 2) {
        const int q = u ? p - nx : p - 1;
        other = C(0.25) * (to_c<C>(src[q]) + to_c<C>(src[q + 1]) + to_c<C>(src[q + nx]) + to_c<C>(src[q + nx + 1]));
        work[p] = from_c<C>(other);
    } else {
        other = to_c<C>(work[p]);
    }
    if (m != 1) return;
    const C mine = to_c<C>(own);
    (u ? a.ru : a.rv)[p] = drag<C>(u ? mine : other, u ? other : mine, D, z0);
}

template <typename C>
__device__ __forceinline__ void momentum_2d_friction_point(const FricArgs& a, int i, int j)
{
    momentum_2d_friction_half<C>(a, 0, i, j);
    momentum_2d_friction_half<C>(a, 1, i, j);
}

// Momentum.coriolis, DEFAULT scheme (momentum.py:1127-1148): interp_xy of the
// transport to the other velocity grid, times f, negated for the V equation.
// (ioff, joff) are the interp_xy offsets: U -> V (1, 0); V -> U (0, 1).
// C: arithmetic (float in the mixed form, whose transport update reads the
// term as a float tendency).
// true where the interpolation writes point (i, j) of the target grid
__device__ __forceinline__ bool coriolis_2d_inside(int nx, int ny, int ioff, int joff, int i, int j)
{
    const int si = i - ioff, sj = j - joff;
    return si >= 0 && sj >= 0 && si <= nx - 2 && sj <= ny - 2;
}

// The term at (i, j) inside the interpolation range; src(i, j) returns the
// transport at a source point.
template <typename C, typename Src>
__device__ __forceinline__ double coriolis_2d_value(int ioff, int joff, int i, int j, const Src& src, double cor,
                                                    int negate)
{
    const int si = i - ioff, sj = j - joff;
    C v = C(0.25) * (to_c<C>(src(si, sj)) + to_c<C>(src(si + 1, sj)) + to_c<C>(src(si, sj + 1)) +
                     to_c<C>(src(si + 1, sj + 1)));
    v = v * to_c<C>(cor);
    return from_c<C>(negate ? -v : v);
}

// ... and outside it (the previous value times f)
template <typename C>
__device__ __forceinline__ double coriolis_2d_outside(double old, double cor, int negate)
{
    C v = to_c<C>(old);
    v = v * to_c<C>(cor);
    return from_c<C>(negate ? -v : v);
}

template <typename C>
__device__ __forceinline__ void coriolis_2d_point(int nx, int ny, int ioff, int joff, const double* src,
                                                  const double* cor, double* out, int negate, int i, int j)
{
    const long long p = (long long)j * nx + i;
    if (coriolis_2d_inside(nx, ny, ioff, joff, i, j)) {
        auto at = [&](int si, int sj) { return src[(long long)sj * nx + si]; };
        out[p] = coriolis_2d_value<C>(ioff, joff, i, j, at, cor[p], negate);
    } else {
        out[p] = coriolis_2d_outside<C>(out[p], cor[p], negate);
    }
}

// Momentum.advance_depth_integrated's transport update (momentum.F90:147-189)
// at interior point p; a: the fields of one direction (U or V).
struct Transport2DArgs {
    const int* mask;
    const double *alpha, *D, *dp, *taus, *cor, *adv, *diff, *damp, *SA, *SB, *SD, *SF, *r;
    double* U;
};

// The operands of one point but the Coriolis term, all loaded before the mask
// is tested (one round of independent loads per point).
struct TransportIn {
    int m;
    double U, SF, D, dp, alpha, taus, adv, diff, damp, SA, SB, SD, r;
};

__device__ __forceinline__ TransportIn transport_2d_load(const Transport2DArgs& a, long long p)
{
    return TransportIn{a.mask[p], a.U[p], a.SF[p], a.D[p], a.dp[p], a.alpha[p], a.taus[p],
                       a.adv[p], a.diff[p], a.damp[p], a.SA[p], a.SB[p], a.SD[p], a.r[p]};
}

// The transport after the update: the new value where the mask is 1, else the
// old one.  cor: the Coriolis term.  MIXED: the tendency is summed in float,
// the transport is updated in double, and the implicit friction factor
// 1/(1 + x), x = dt r / D, is applied as U - U x/(1 + x) with the small
// correction in float (no FP64 division).
template <bool MIXED>
__device__ __forceinline__ double transport_2d_value(const TransportIn& a, double dt, double cor)
{
    if (a.m != 1) return a.U;
    if constexpr (!MIXED) {
        const double rho0i = 1.0 / GETM_RHO0;
        const double Slr = getm_positive_i(a.U) ? getm_fmin_i(a.SF, 0.0) : getm_fmax_i(a.SF, 0.0);
        // (contracted in one way in every kernel that forms it)
        const double sum = __fma_rn(a.taus, rho0i, cor) + a.adv + a.diff + a.damp + a.SA + a.SB + a.SD + Slr;
        const double tend = __fma_rn(a.alpha, sum, __dmul_rn(__dmul_rn(-GETM_G, a.D), a.dp));
        // (U + dt tend) / (1 + dt r / D) with one division
        return getm_div(__dmul_rn(__fma_rn(dt, tend, a.U), a.D), __fma_rn(dt, a.r, a.D));
    } else {
        const float rho0i = (float)(1.0 / GETM_RHO0);
        const float sf = getm_d2f_approx(a.SF);
        const float Slr = getm_positive_i(a.U) ? fminf(sf, 0.f) : fmaxf(sf, 0.f);
        const float Dp = getm_d2f_approx(a.D);
        const float dtf = (float)dt;
        const float tend = -(float)GETM_G * Dp * getm_d2f_approx(a.dp) +
                           getm_d2f_approx(a.alpha) *
                               (getm_d2f_approx(a.taus) * rho0i + getm_d2f_approx(cor) + getm_d2f_approx(a.adv) +
                                getm_d2f_approx(a.diff) + getm_d2f_approx(a.damp) + getm_d2f_approx(a.SA) +
                                getm_d2f_approx(a.SB) + getm_d2f_approx(a.SD) + Slr);
        const double num = a.U + getm_f2d(dtf * tend);
        const float x = dtf * getm_d2f_approx(a.r) / Dp;
        return num - getm_f2d(getm_d2f_approx(num) * (x / (1.f + x)));
    }
}

template <bool MIXED>
__device__ __forceinline__ void transport_2d_point(const Transport2DArgs& a, double dt, long long p)
{
    const double cor = a.cor[p];
    const TransportIn in = transport_2d_load(a, p);
    if (in.m == 1) a.U[p] = transport_2d_value<MIXED>(in, dt, cor);
}

// _U_cum += U; _V_cum += V (momentum.py:716-718), every point
__device__ __forceinline__ void accumulate_2d_point(const double* U, const double* V, double* Uc, double* Vc,
                                                    long long p)
{
    Uc[p] = Uc[p] + U[p];
    Vc[p] = Vc[p] + V[p];
}

// zo = z (every point), then the surface elevation update
// (simulation.py:1468-1486 -> wrapper.F90:496-523)
// the elevation update at an interior water point (wrapper.F90:496-523),
// contracted in one way in every kernel that forms it
__device__ __forceinline__ double elevation_new(double zp, double dt, double Uw, double dyw, double Ue, double dye,
                                                double Vs, double dxs, double Vn, double dxn, double ia, double fw)
{
    const double t = __fma_rn(-Vn, dxn, __fma_rn(Vs, dxs, __fma_rn(Uw, dyw, -__dmul_rn(Ue, dye))));
    return __fma_rn(dt, __fma_rn(t, ia, fw), zp);
}

__device__ __forceinline__ void surface_elevation_fused_point(int nx, int ny, int halox, int haloy, const int* mask,
                                                              const double* dyu, const double* dxv,
                                                              const double* iarea, double* z, double* zo,
                                                              const double* U, const double* V, const double* fwf,
                                                              double dt, int i, int j)
{
    const long long p = (long long)j * nx + i;
    const double zp = z[p];
    zo[p] = zp;
    if (i < halox || i >= nx - halox || j < haloy || j >= ny - haloy) return;
    // every operand is loaded before the mask is tested
    const int m = mask[p];
    const double Uw = U[p - 1], dyw = dyu[p - 1], Ue = U[p], dye = dyu[p], Vs = V[p - nx], dxs = dxv[p - nx];
    const double Vn = V[p], dxn = dxv[p], ia = iarea[p], fw = fwf[p];
    if (m != 1) return;
    z[p] = elevation_new(zp, dt, Uw, dyw, Ue, dye, Vs, dxs, Vn, dxn, ia, fw);
}


// reconstruct_transport_change (momentum.F90:323-340) at point p of a row
// inside jmin..jmax (T: type of un and Uo)
template <typename T>
__device__ __forceinline__ void reconstruct_point(T* un, const double* hn, const T* Uo, double idt, long long p)
{
    if constexpr (std::is_same<T, double>::value) un[p] = (un[p] * hn[p] - Uo[p]) * idt;
    else un[p] = (un[p] * getm_d2f_approx(hn[p]) - Uo[p]) * (T)idt;
}

// surface_pressure_gradient (wrapper.F90:525-565) at interior point (i, j)
struct SpgArgs {
    int nx;
    const int *umask, *vmask;
    const double *idxu, *idyv, *z, *sp, *H, *D;
    double Dmin;
    double *dpdx, *dpdy;
};

// MIXED: the elevation bounds on the integer pipe, the two differences in
// FP64 and the rest in float (the mixed transport update reads the gradient
// as a float).
// The bound -H + min(Dmin, D) of an elevation, H at one point and D at its
// neighbour; dry = -H + Dmin, which it is wherever the neighbour is deeper
// than Dmin (the sum is formed out of line elsewhere, so that it costs nothing).
static __device__ __noinline__ double spg_shallow(double H, double m) { return -H + m; }

__device__ __forceinline__ double spg_bound(double dry, double H, double Dmin, double D)
{
    const double m = getm_fmin_i(Dmin, D);
    return __double_as_longlong(m) == __double_as_longlong(Dmin) ? dry : spg_shallow(H, m);
}

// One direction's gradient out (mask m): z, H, D, sp and B = -H + Dmin at the
// point (0) and its neighbour (1)
template <bool MIXED>
__device__ __forceinline__ void spg_half(double* out, double Dmin, long long p, int m, double z0, double z1, double H0,
                                         double H1, double D0, double D1, double B0, double B1, double sp0, double sp1,
                                         double id)
{
    if (m != 1) return;
    const double zp = getm_fmax_i(z1, spg_bound(B0, H0, Dmin, D1));
    const double zm = getm_fmax_i(z0, spg_bound(B1, H1, Dmin, D0));
    if constexpr (MIXED) {
        const float gi = (float)(1.0 / (GETM_G * GETM_RHO0));
        const float g = getm_d2f_approx(zp - zm) + getm_d2f_approx(sp1 - sp0) * gi;
        out[p] = getm_f2d(g * getm_d2f_approx(id));
    } else {
        const double gammai = 1.0 / (GETM_G * GETM_RHO0);
        out[p] = (zp - zm + (sp1 - sp0) * gammai) * id;
    }
}

template <bool MIXED = false>
__device__ __forceinline__ void spg_point(const SpgArgs& a, long long p)
{
    const long long n = p + a.nx;
    // every operand is loaded before the masks are tested
    const int mu = a.umask[p], mv = a.vmask[p];
    const double z0 = a.z[p], z1 = a.z[p + 1], zn = a.z[n], H0 = a.H[p], H1 = a.H[p + 1], Hn = a.H[n];
    const double D0 = a.D[p], D1 = a.D[p + 1], Dn = a.D[n], sp0 = a.sp[p], sp1 = a.sp[p + 1], spn = a.sp[n];
    const double idx = a.idxu[p], idy = a.idyv[p], B0 = -H0 + a.Dmin;
    spg_half<MIXED>(a.dpdx, a.Dmin, p, mu, z0, z1, H0, H1, D0, D1, B0, -H1 + a.Dmin, sp0, sp1, idx);
    spg_half<MIXED>(a.dpdy, a.Dmin, p, mv, z0, zn, H0, Hn, D0, Dn, B0, -Hn + a.Dmin, sp0, spn, idy);
}

// interp_x / interp_y (interpolation.F90:9-40) of one point: t = mean of s
// at p and its neighbour at +step, stored at p + off (off = 0 or step)
template <typename T>
__device__ __forceinline__ void interp_pair_point(const T* s, T* t, long long p, long long step, long long off)
{
    if constexpr (std::is_same<T, double>::value) t[p + off] = getm_half(s[p] + s[p + step]);
    else t[p + off] = T(0.5) * (s[p] + s[p + step]);
}
