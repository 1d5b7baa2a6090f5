// Horizontal advection passes as device functions (shared by the one-pass
// kernels of advection.cu and the fused 2D-substep kernel of split2d.cu).
// Reference: src/operators/advection_schemes/advection.F90.template
// (u2d :23-121, v2d :123-221) and limiters.h.
#pragma once

#include "getm_common.cuh"

#define GETM_MAX_BATCH 32

// ---------------------------------------------------------------------------
// horizontal pass kernels
// ---------------------------------------------------------------------------
// T is the type of the advected fields, V that of the velocities (T unless
// given): double for the FP64 form, float for the mixed form; the mixed form
// with FP64 tracer storage has T = double, V = float (its increments are
// still formed in float).  Layer thicknesses and all grid metrics are double
// in every form.
template <typename T, typename V = T>
struct HPassArgs {
    int nx_, ny_, nk;
    long long plane;            // nx_ * ny_
    int ilo, ihi, jlo, jhi;     // C interior bounds (inclusive) of the T grid
    const int* umask;           // mask of the velocity grid of this direction
    const double* idx;          // x: idx of U grid; y: idy of V grid (Courant number)
    const double* dy;           // x: dy of U grid;  y: dx of V grid (face length)
    const int* tmask;
    const double* iA;
    const double* Ah;           // 2D horizontal diffusivity on the velocity grid, or NULL
    const V* u;                 // velocity (nk layers)
    const double* hu;           // layer thickness on the velocity grid (nk layers)
    const double* h_in;
    double* h_out;
    double dt;
    int scheme;
    int ntracer;
    // mixed form: float copies of dt and of the metrics above; increment != 0
    // selects float increments for double fields (2D momentum)
    int increment;
    float dtf;
    int ych;                    // rows a warp marches in the 3D y pass (launch-shape knob)
    const float* idx_f;
    const float* dy_f;
    const float* iA_f;
    const T* fin[GETM_MAX_BATCH];
    T* fout[GETM_MAX_BATCH];
};

// Epilogue of a pass: called once per updated (or copied) cell with the
// cell's flat index p3, its row j, the new value of the first field and the
// new thickness.  The default does nothing; the 2D substep uses
// it to form the momentum advection term as each cell is finished.
struct NoEpi {
    __device__ __forceinline__ void operator()(long long, int, double, double) const {}
};

// ---------------------------------------------------------------------------
// Increment form of the passes (template :61-116).
//
// With hold - hnew = dt iA (QU_e - QU_w), the reference update
// (hold f - dt iA (QU_e f_e - QU_w f_w)) / hnew equals
//     f - dt iA (QU_e (f_e - f) - QU_w (f_w - f)) / hnew
// exactly, where f_e, f_w are the limited face values.  Each face therefore
// provides el = QU (face - left cell) and er = QU (face - right cell), formed
// from differences of neighbouring values, so rounding scales with the change
// of the field and a field at rest is reproduced exactly.
//
// C: the arithmetic of the increments.
// * C = float (mixed form): float32 rounding scales with the change, and the
//   only FP64 operations per cell are the thickness update hnew = hold - dh
//   and, for fields stored in double, the difference and the final sum.
// * C = double (FP64 form): GB300 issues an FP64 instruction at 1/64 of the
//   float rate, so the number of FP64 instructions is the time of the pass.
//   In increment form and with the division-free limiter on the integer pipe
//   a cell takes 13 of them for the geometry and the thickness and 6 per
//   field (superbee); the reference's order of evaluation took about 120 for
//   one field, two thirds of them in its two divisions per field and in the
//   extra face of each warp's first lane (or tile's first row).  Measured, us
//   per pass: 120 x 100 x 30, one field, superbee, x 93.6 -> 27.5, y 97.2 ->
//   28.5; 173 x 131 x 23, six fields, HSIMT and diffusion, x 446 -> 118, y 428
//   -> 132 (FP64 pipe 77 % busy).  Against quad precision the five-pass split's
//   error falls from 2.0e-16 to 1.3e-16 (a result is rounded once per pass,
//   not three times).  Products and sums are rounded as written (intrinsics,
//   no contraction): the separate passes and the 2D substep share
//   these functions and give the same bits.
// ---------------------------------------------------------------------------
// Storage type S of the advected field and V of the velocities: float (the
// 3D fields of the mixed form) or double (with C = float: the 2D
// depth-averaged momentum and the tracers of the mixed form, whose state
// stays FP64 while its increments are evaluated in float).  Differences of
// neighbouring values are formed in S and then narrowed to C, so they keep
// their accuracy when the values are close.

// a value or a difference in S (or V) narrowed to the arithmetic type
template <typename C, typename S>
__device__ __forceinline__ C hx_c(S x)
{
    if constexpr (std::is_same<C, double>::value) return (double)x;
    else return inc_f<S>(x);
}

// the metrics and the time step in the arithmetic type
template <typename C, typename S, typename V>
__device__ __forceinline__ const C* hx_dy(const HPassArgs<S, V>& a)
{
    if constexpr (std::is_same<C, double>::value) return a.dy;
    else return a.dy_f;
}

template <typename C, typename S, typename V>
__device__ __forceinline__ const C* hx_idx(const HPassArgs<S, V>& a)
{
    if constexpr (std::is_same<C, double>::value) return a.idx;
    else return a.idx_f;
}

template <typename C, typename S, typename V>
__device__ __forceinline__ const C* hx_iA(const HPassArgs<S, V>& a)
{
    if constexpr (std::is_same<C, double>::value) return a.iA;
    else return a.iA_f;
}

template <typename C, typename S, typename V>
__device__ __forceinline__ C hx_dt(const HPassArgs<S, V>& a)
{
    if constexpr (std::is_same<C, double>::value) return a.dt;
    else return a.dtf;
}

__device__ __forceinline__ float hx_mul3(float x, float y, float z) { return x * y * z; }
__device__ __forceinline__ double hx_mul3(double x, double y, double z) { return __dmul_rn(__dmul_rn(x, y), z); }
__device__ __forceinline__ float hx_abs(float x) { return fabsf(x); }
__device__ __forceinline__ double hx_abs(double x) { return fabs(x); }
__device__ __forceinline__ bool hx_positive(float x) { return x > 0.f; }
__device__ __forceinline__ bool hx_positive(double x) { return getm_positive_i(x); }
__device__ __forceinline__ float hx_ahd(float ah, float hu, float idx, float dy) { return -ah * hu * idx * dy; }
__device__ __forceinline__ double hx_ahd(double ah, double hu, double idx, double dy)
{
    return -__dmul_rn(hx_mul3(ah, hu, idx), dy);
}

// thickness of an updated cell and dt iA / hnew
__device__ __forceinline__ void hx_cell(float dt, float QUe, float QUw, float iA, double hold, double& hnew,
                                        float& coef)
{
    const float dh = dt * (QUe - QUw) * iA;
    hnew = hold - getm_f2d(dh);
    coef = dt * iA / (getm_d2f_approx(hold) - dh);
}

__device__ __forceinline__ void hx_cell(double dt, double QUe, double QUw, double iA, double hold, double& hnew,
                                        double& coef)
{
    const double c = __dmul_rn(dt, iA);
    hnew = __fma_rn(-c, __dadd_rn(QUe, -QUw), hold);
    coef = __dmul_rn(c, getm_rcp(hnew));
}

// el and er of an active face, given d = f[b] - f[a] across the face and the
// differences on either side, dprev = f[a] - f[a-1] and dnext = f[b+1] - f[b];
// tf: the face's limiter constants; ahd = -Ah hu idx dy (diff: whether there
// is horizontal diffusion).  The limiter is odd in its two differences, so the
// side away from the flow is selected first and one evaluation serves both
// flow directions.
__device__ __forceinline__ void hx_face(const TvdFace<float>& tf, bool up, bool uu_ok, float QU, float dprev, float d,
                                        float dnext, float ahd, bool, float& el, float& er)
{
    const float lim = getm_tvd_dev_c(tf, d, uu_ok ? (up ? dprev : dnext) : 0.f);
    const float dev = up ? lim : -lim;
    const float fd = ahd * d;
    el = QU * (up ? dev : d + dev) + fd;
    er = QU * (up ? dev - d : dev) + fd;
}

// FP64: with G = QU 0.5 (1 - cfl) phi(r) d and P = QU d, the upwind side's
// value is +-G (+ the diffusive flux) and the other's differs from it by P:
// four FP64 instructions with the product for G's first factor formed once
// per face (tf.half1mc holds it).
__device__ __forceinline__ void hx_face(const TvdFace<double>& tf, bool up, bool uu_ok, double QU, double dprev,
                                        double d, double dnext, double ahd, bool diff, double& el, double& er)
{
    double G = getm_negate_if(__dmul_rn(tf.half1mc, getm_tvd_phi(tf, QU, d, uu_ok ? (up ? dprev : dnext) : 0.0)), !up);
    if (diff) G = __fma_rn(ahd, d, G);
    const double other = __dadd_rn(G, getm_negate_if(__dmul_rn(QU, d), up));
    el = up ? G : other;
    er = up ? other : G;
}

// the face's limiter constants
__device__ __forceinline__ TvdFace<float> hx_tvd(int scheme, float cfl, float) { return getm_tvd_face_c(scheme, cfl); }

__device__ __forceinline__ TvdFace<double> hx_tvd(int scheme, double cfl, double QU)
{
    TvdFace<double> tf = getm_tvd_face_c(scheme, cfl);
    tf.half1mc = __dmul_rn(QU, tf.half1mc);
    return tf;
}

// the new value of a field in a cell: el_e of its east (north) face, er_w of
// its west (south) face
template <typename S>
__device__ __forceinline__ S hx_new(S f, float coef, float el_e, float er_w)
{
    return inc_add<S>(f, -coef * (el_e - er_w));
}

__device__ __forceinline__ double hx_new(double f, double coef, double el_e, double er_w)
{
    return __fma_rn(-coef, __dadd_rn(el_e, -er_w), f);
}

// x-direction pass in increment form.  A warp owns one row segment: lane L
// computes the face at U point a = i0 - 1 + L (between cells a and a+1) and,
// for L < 31, updates cell a + 1, whose east face comes from lane L + 1 by a
// shuffle; segments therefore advance by 31 cells.  Every lane runs the same
// instructions (no per-lane special paths): each field is read with one
// coalesced load per warp plus one load of the three values just outside
// the segment (lanes 0-2), and all loads of a lane are independent.
constexpr int HX_STRIDE = 31;

// KB layers k0 .. k0+KB-1 (those below nk) of row j: the 2D fields (masks,
// metrics) are loaded once for all of them, and every load of the KB layers
// is issued before any value is used.
template <typename S, int KB, typename Epi = NoEpi, typename V = S, typename C = float>
__device__ __forceinline__ void hpass_x_inc_rows(const HPassArgs<S, V>& a, int bx, int j, int k0, int lane,
                                                 const Epi& epi = Epi())
{
    constexpr unsigned FULL = 0xffffffffu;
    const int i0 = bx * HX_STRIDE;
    const int ia = i0 - 1 + lane;  // this lane's face (U point) and its west cell
    const int ib = ia + 1;         // the cell this lane updates (lanes 0-30)
    const long long r2 = (long long)j * a.nx_;
    const bool jrow = j >= a.jlo && j <= a.jhi;
    const bool ain = ia >= 0 && ia < a.nx_;
    // lanes 0-2 address the points i0-2, i0+31, i0+32 just outside the lanes' range
    const int ix = lane == 0 ? i0 - 2 : i0 + 30 + lane;
    const bool xin = lane < 3 && ix >= 0 && ix < a.nx_;
    const bool bin = lane < HX_STRIDE && ib < a.nx_;
    // in-bounds copies of the indices for the loads
    const int iac = min(max(ia, 0), a.nx_ - 1), ixc = min(max(ix, 0), a.nx_ - 1), ibc = min(ib, a.nx_ - 1);
    const int um_raw = a.umask[r2 + iac];
    const int umx_raw = a.umask[r2 + ixc];
    const C dyf = hx_dy<C>(a)[r2 + iac], idxf = hx_idx<C>(a)[r2 + iac];
    const C ahraw = a.Ah ? hx_c<C>(a.Ah[r2 + iac]) : C(0);
    const int tm = a.tmask[r2 + ibc];
    const C iaf = hx_iA<C>(a)[r2 + ibc];
    V uraw[KB];
    double huraw[KB], hold[KB];
#pragma unroll
    for (int kk = 0; kk < KB; kk++) {
        const long long r3 = (long long)min(k0 + kk, a.nk - 1) * a.plane + r2;
        uraw[kk] = a.u[r3 + iac];
        huraw[kk] = a.hu[r3 + iac];
        hold[kk] = a.h_in[r3 + ibc];
    }
    const int ntg = a.ntracer < 2 ? a.ntracer : 2;  // tracers of the first group
    S fa_[KB][2], fx_[KB][2];
#pragma unroll
    for (int kk = 0; kk < KB; kk++) {
        const long long r3 = (long long)min(k0 + kk, a.nk - 1) * a.plane + r2;
#pragma unroll
        for (int q = 0; q < 2; q++) {
            if (q < ntg) {
                const S* __restrict__ f = a.fin[q] + r3;
                fa_[kk][q] = f[iac];
                fx_[kk][q] = f[ixc];
            } else {
                fa_[kk][q] = S(0);
                fx_[kk][q] = S(0);
            }
        }
    }

    // face masks (the same for every layer)
    const bool f_in = ain && jrow && ia >= a.ilo - 1 && ia <= a.ihi;
    const int um = ain ? um_raw : 0;
    const int umx = xin ? umx_raw : 0;
    int um_w = __shfl_up_sync(FULL, um, 1), um_e = __shfl_down_sync(FULL, um, 1);
    const int umx0 = __shfl_sync(FULL, umx, 0), umx1 = __shfl_sync(FULL, umx, 1);
    if (lane == 0) um_w = umx0;
    if (lane == 31) um_e = umx1;
    const bool act = f_in && getm_flux_point(um);
    const bool upd = bin && jrow && ib >= a.ilo && ib <= a.ihi && tm == 1;

#pragma unroll
    for (int kk = 0; kk < KB; kk++) {
        if (k0 + kk >= a.nk) break;
        const long long r3 = (long long)(k0 + kk) * a.plane + r2;
        C QU = C(0), cfl = C(0), ahd = C(0);
        bool up = false, uu_ok = false;
        if (act) {
            const C uu = hx_c<C>(uraw[kk]);
            const C huf = hx_c<C>(huraw[kk]);
            QU = hx_mul3(uu, huf, dyf);
            cfl = hx_abs(hx_mul3(uu, hx_dt<C>(a), idxf));
            up = hx_positive(uu);
            uu_ok = getm_flux_point(up ? um_w : um_e);
            if (a.Ah) ahd = hx_ahd(ahraw, huf, idxf, dyf);
        }
        const C QUe = __shfl_down_sync(FULL, QU, 1);  // east face of cell ib

        // thickness update of cell ib
        C coef = C(0);  // dt iA / hnew
        double hnew = hold[kk];
        if (bin) {
            if (upd) hx_cell(hx_dt<C>(a), QUe, QU, iaf, hold[kk], hnew, coef);
            a.h_out[r3 + ib] = hnew;
        }
        const TvdFace<C> tf = hx_tvd(a.scheme, cfl, QU);
        // tracers two at a time (the first two preloaded with the layer)
        for (int t = 0; t < a.ntracer; t += 2) {
            const int nt = a.ntracer - t >= 2 ? 2 : 1;
            S fa2[2], fx2[2];
            if (t == 0) {
                fa2[0] = fa_[kk][0]; fa2[1] = fa_[kk][1];
                fx2[0] = fx_[kk][0]; fx2[1] = fx_[kk][1];
            } else {
#pragma unroll
                for (int q = 0; q < 2; q++) {
                    const S* __restrict__ f = a.fin[t + (q < nt ? q : 0)] + r3;
                    fa2[q] = f[iac];
                    fx2[q] = f[ixc];
                }
            }
#pragma unroll
            for (int q = 0; q < 2; q++) {
                if (q >= nt) break;
                const S fa = ain ? fa2[q] : S(0);
                const S fx = xin ? fx2[q] : S(0);
                S fb = __shfl_down_sync(FULL, fa, 1);  // f[ia+1]
                const S x0 = __shfl_sync(FULL, fx, 0), x1 = __shfl_sync(FULL, fx, 1), x2 = __shfl_sync(FULL, fx, 2);
                if (lane == 31) fb = x1;
                const C d = hx_c<C>(fb - fa);
                C dprev = __shfl_up_sync(FULL, d, 1), dnext = __shfl_down_sync(FULL, d, 1);
                // the two differences the shuffles cannot supply, in one operation
                const C e = hx_c<C>(lane == 0 ? fa - x0 : x2 - x1);
                if (lane == 0) dprev = e;
                if (lane == 31) dnext = e;
                // el = QU (face - f[ia]) (east side of cell ia), er = QU (face - f[ib])
                C el = C(0), er = C(0);
                if (act) hx_face(tf, up, uu_ok, QU, dprev, d, dnext, ahd, a.Ah != nullptr, el, er);
                const C el_e = __shfl_down_sync(FULL, el, 1);  // east face of cell ib, seen from ib
                if (bin) {
                    const S fn = upd ? hx_new(fb, coef, el_e, er) : fb;
                    a.fout[t + q][r3 + ib] = fn;
                    if (t + q == 0) epi(r3 + ib, j, (double)fn, hnew);
                }
            }
        }
    }
}

// x pass in increment form with four cells per lane, for the 3D passes.  A
// warp sweeps nrow rows of a layer from west to east, one behind the other, in
// chunks of 128 cells; lane L of a chunk owns four cells and their east faces,
// so every load and store of the lane is one 16-byte vector (two for doubles)
// at an aligned address (the caller checks nx_ % 4 == 0 and the pointers'
// alignment).  Rows are contiguous, so a chunk may end one row and begin the
// next: with at least two halo cells no face or cell that is used looks across
// that seam, and only a warp's last chunk has idle lanes (a 404-cell row by
// itself fills 3.2 of its 4 chunks: 400 x 300 x 40, two FP64-stored tracers, 119 ->
// 104 us, a float field 60 -> 55 us).  A face needs the values of the lanes
// beside it (shuffles), the chunk to the west hands its last face over in
// registers, and the last lane reads the two cells east of the chunk.  Each difference
// of neighbouring values is formed once (it serves the face and, in the
// limiter, both faces beside it: one FP64 subtraction per cell and field
// instead of two for FP64 storage).  Every face and cell is evaluated with
// the same expressions as hpass_x_inc_rows, so both give the same bits.
// Fields t0 and t0 + 1 are swept together (the thickness is written with the
// first), further pairs by warps of their own.
template <typename T>
__device__ __forceinline__ void xv_load4(const T* p, T (&o)[4])
{
    if constexpr (sizeof(T) == 8) {
        const double2 a = *reinterpret_cast<const double2*>(p);
        const double2 b = *reinterpret_cast<const double2*>(p + 2);
        o[0] = a.x; o[1] = a.y; o[2] = b.x; o[3] = b.y;
    } else if constexpr (std::is_same<T, int>::value) {
        const int4 a = *reinterpret_cast<const int4*>(p);
        o[0] = a.x; o[1] = a.y; o[2] = a.z; o[3] = a.w;
    } else {
        const float4 a = *reinterpret_cast<const float4*>(p);
        o[0] = a.x; o[1] = a.y; o[2] = a.z; o[3] = a.w;
    }
}

template <typename T>
__device__ __forceinline__ void xv_store4(T* p, const T (&v)[4])
{
    if constexpr (sizeof(T) == 8) {
        *reinterpret_cast<double2*>(p) = make_double2(v[0], v[1]);
        *reinterpret_cast<double2*>(p + 2) = make_double2(v[2], v[3]);
    } else {
        *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
    }
}

template <typename S, typename V = S>
__device__ __forceinline__ void hpass_x_vec_rows(const HPassArgs<S, V>& a, int j0, int nrow, int k, int lane, int t0)
{
    constexpr unsigned FULL = 0xffffffffu;
    const int nx = a.nx_;
    const int nq = nx / 4;  // quads of cells per row
    const int total = nq * nrow;
    const long long r2 = (long long)j0 * nx;
    const long long r3 = (long long)k * a.plane + r2;
    const int nt = a.ntracer - t0 >= 2 ? 2 : a.ntracer - t0;  // 0 with no fields
    // the west face of the chunk's first cell: the chunk to the west's
    // last face (nothing west of the rows: an inactive face)
    float cQU = 0.f;
    int cum = 0;
    float cd[2] = {0.f, 0.f}, cer[2] = {0.f, 0.f};
    int row = lane / nq, iq = lane - row * nq;  // the lane's row and quad
    for (int q0 = 0; q0 < total; q0 += 32) {
        const int ib = 4 * (q0 + lane);  // the lane's first cell, from the first row's start
        const int ic = 4 * iq;           // ... in its row
        const bool lin = q0 + lane < total;  // all four cells or none
        const int ie = 4 * (q0 + 32);        // the first cell east of the chunk
        const bool ein = q0 + 32 < total;
        const int j = j0 + row;
        const bool jrow = j >= a.jlo && j <= a.jhi;
        int um[4] = {0, 0, 0, 0}, tm[4] = {0, 0, 0, 0};
        float dyf[4] = {0.f, 0.f, 0.f, 0.f}, idxf[4] = {0.f, 0.f, 0.f, 0.f}, iaf[4] = {0.f, 0.f, 0.f, 0.f};
        float ahraw[4] = {0.f, 0.f, 0.f, 0.f};
        V uraw[4] = {V(0), V(0), V(0), V(0)};
        double huraw[4] = {0.0, 0.0, 0.0, 0.0}, hold[4] = {0.0, 0.0, 0.0, 0.0};
        if (lin) {
            xv_load4(a.umask + r2 + ib, um);
            xv_load4(a.tmask + r2 + ib, tm);
            xv_load4(a.dy_f + r2 + ib, dyf);
            xv_load4(a.idx_f + r2 + ib, idxf);
            xv_load4(a.iA_f + r2 + ib, iaf);
            xv_load4(a.u + r3 + ib, uraw);
            xv_load4(a.hu + r3 + ib, huraw);
            xv_load4(a.h_in + r3 + ib, hold);
            if (a.Ah) {
                double ah[4];
                xv_load4(a.Ah + r2 + ib, ah);
#pragma unroll
                for (int m = 0; m < 4; m++) ahraw[m] = getm_d2f_approx(ah[m]);
            }
        }
        // masks of the velocity points beside the lane's first and last faces
        int umW = __shfl_up_sync(FULL, um[3], 1), umE = __shfl_down_sync(FULL, um[0], 1);
        if (lane == 0) umW = cum;
        if (lane == 31) umE = ein ? a.umask[r2 + ie] : 0;

        // face geometry (the same expressions as hpass_x_inc_rows)
        float QU[4], cfl[4], ahd[4];
        bool up[4], uu_ok[4], act[4];
#pragma unroll
        for (int m = 0; m < 4; m++) {
            const int ia = ic + m;
            const bool f_in = lin && jrow && ia >= a.ilo - 1 && ia <= a.ihi;
            act[m] = f_in && getm_flux_point(um[m]);
            QU[m] = 0.f; cfl[m] = 0.f; ahd[m] = 0.f;
            up[m] = false; uu_ok[m] = false;
            if (act[m]) {
                const float uu = inc_f<V>(uraw[m]);
                const float huf = getm_d2f_approx(huraw[m]);
                QU[m] = uu * huf * dyf[m];
                cfl[m] = fabsf(uu * a.dtf * idxf[m]);
                up[m] = uu > 0.f;
                const int mw = m > 0 ? um[m - 1] : umW, me = m < 3 ? um[m + 1] : umE;
                uu_ok[m] = getm_flux_point(up[m] ? mw : me);
                if (a.Ah) ahd[m] = -ahraw[m] * huf * idxf[m] * dyf[m];
            }
        }
        float QUw0 = __shfl_up_sync(FULL, QU[3], 1);  // west face of the lane's first cell
        if (lane == 0) QUw0 = cQU;

        // thickness update of the lane's cells
        float coef[4];
        bool upd[4];
        double hnew[4];
#pragma unroll
        for (int m = 0; m < 4; m++) {
            const int c = ic + m;
            upd[m] = lin && jrow && c >= a.ilo && c <= a.ihi && tm[m] == 1;
            coef[m] = 0.f;
            hnew[m] = hold[m];
            if (upd[m]) {
                const float QUw = m > 0 ? QU[m - 1] : QUw0;
                hx_cell(a.dtf, QU[m], QUw, iaf[m], hold[m], hnew[m], coef[m]);
            }
        }
        if (t0 == 0 && lin) xv_store4(a.h_out + r3 + ib, hnew);

#pragma unroll
        for (int q = 0; q < 2; q++) {
            if (q >= nt) break;
            const S* __restrict__ f = a.fin[t0 + q] + r3;
            S fv[4] = {S(0), S(0), S(0), S(0)};
            if (lin) xv_load4(f + ib, fv);
            S fE0 = S(0), fE1 = S(0);  // the two cells east of the chunk (last lane)
            if (lane == 31) {
                if (ein) { fE0 = f[ie]; fE1 = f[ie + 1]; }
            }
            S fn0 = __shfl_down_sync(FULL, fv[0], 1);
            if (lane == 31) fn0 = fE0;
            // differences of neighbouring values in the storage type, then
            // narrowed (d[m]: across face m)
            float d[4];
            d[0] = inc_f<S>(fv[1] - fv[0]);
            d[1] = inc_f<S>(fv[2] - fv[1]);
            d[2] = inc_f<S>(fv[3] - fv[2]);
            d[3] = inc_f<S>(fn0 - fv[3]);
            float dW = __shfl_up_sync(FULL, d[3], 1), dE = __shfl_down_sync(FULL, d[0], 1);
            if (lane == 0) dW = cd[q];
            if (lane == 31) dE = inc_f<S>(fE1 - fE0);
            float el[4], er[4];
#pragma unroll
            for (int m = 0; m < 4; m++) {
                el[m] = 0.f; er[m] = 0.f;
                if (act[m]) {
                    const TvdFace<float> tf = getm_tvd_face_c(a.scheme, cfl[m]);
                    const float dprev = m > 0 ? d[m - 1] : dW, dnext = m < 3 ? d[m + 1] : dE;
                    hx_face(tf, up[m], uu_ok[m], QU[m], dprev, d[m], dnext, ahd[m], a.Ah != nullptr, el[m], er[m]);
                }
            }
            float erW = __shfl_up_sync(FULL, er[3], 1);  // west face of the lane's first cell
            if (lane == 0) erW = cer[q];
            S out[4];
#pragma unroll
            for (int m = 0; m < 4; m++) {
                const float ew = m > 0 ? er[m - 1] : erW;
                out[m] = upd[m] ? hx_new(fv[m], coef[m], el[m], ew) : fv[m];
            }
            if (lin) xv_store4(a.fout[t0 + q] + r3 + ib, out);
            cd[q] = __shfl_sync(FULL, d[3], 31);
            cer[q] = __shfl_sync(FULL, er[3], 31);
        }
        cQU = __shfl_sync(FULL, QU[3], 31);
        cum = __shfl_sync(FULL, um[3], 31);
        for (iq += 32; iq >= nq; iq -= nq) row++;
    }
}

// One row (layer k, row j) of the x pass: row = k ny_ + j.
template <typename S, typename Epi = NoEpi, typename V = S, typename C = float>
__device__ __forceinline__ void hpass_x_inc_body(const HPassArgs<S, V>& a, int bx, long long row, int lane,
                                                 const Epi& epi = Epi())
{
    if (row >= (long long)a.ny_ * a.nk) return;  // whole warp shares one row
    const int k = (int)(row / a.ny_);
    const int j = (int)(row - (long long)k * a.ny_);
    hpass_x_inc_rows<S, 1, Epi, V, C>(a, bx, j, k, lane, epi);
}

// y-direction pass in increment form: the transpose of hpass_x_inc_kernel.
// A block of 32 x HY_BY threads covers 32 columns; thread row ty computes the
// face at V point ja = j0 - 1 + ty and, for ty < HY_BY - 1, updates cell
// ja + 1, whose north face comes from thread row ty + 1 through shared
// memory; blocks therefore advance by HY_BY - 1 rows.  The rows of each
// tracer a block needs are staged in shared memory once (one coalesced load
// per row), so every value is read from global memory once per block.
constexpr int HY_BY = 16;
constexpr int HY_STRIDE = HY_BY - 1;

// Rows of a block (one of them the edge) for `tiles` columns of blocks of 32 cells
// over ny rows: 4, so that a plane spreads evenly over the SMs (an FP64 pass
// takes as long as its fullest SM), or 16 (FP64) where that leaves every SM a few
// blocks all the same, for 16 rows repeat less at the edges.  us with 16 / 8 / 4
// rows, FP64 2D advection 97 x 75 22.8 / 18.7 / 18.7, 400 x 300 37.2 / 37.6 / 37.6;
// 2D substep FP64 64 x 64 38.6 / 33.0 / 30.6, 220 x 160 54.4 / 57.4 / 52.5, mixed
// 400 x 300 48.6 / 47.6 / 47.0.  16 also where a grid's 65535 blocks of 4 rows do
// not reach.
inline int hpass_y_rows(long long tiles, int ny, bool f64)
{
    return (f64 && tiles * ((ny + 15) / 15) > 2 * GETM_SMS) || ny >= 3 * 65535 ? 16 : 4;
}

template <typename S, typename C = float, int BY = HY_BY>
struct YIncSmem {
    S sf[BY + 3][32];       // rows j0-2 .. j0+BY
    C sd[BY + 2][32];      // differences f[j+1] - f[j], rows j0-2 .. j0+BY-1
    C sx[BY][32];           // per-face exchange (QU, then el)
};

template <typename S, typename Epi = NoEpi, typename V = S, typename C = float, int BY = HY_BY>
__device__ __forceinline__ void hpass_y_inc_body(const HPassArgs<S, V>& a, int bx, int by, int k, int tx, int ty,
                                                 YIncSmem<S, C, BY>& sm, const Epi& epi = Epi())
{
    auto& sf = sm.sf;
    auto& sd = sm.sd;
    auto& sx = sm.sx;
    const int i = bx * 32 + tx;
    const int j0 = by * (BY - 1);
    const int ja = j0 - 1 + ty;  // this thread's face (V point) and its south cell
    const int jb = ja + 1;       // the cell this thread updates (ty < (BY - 1))
    const long long s = a.nx_;
    const long long base = (long long)k * a.plane + i;  // + j * s
    const bool icol = i < a.nx_;
    const bool ain = icol && ja >= 0 && ja < a.ny_;
    const bool iint = i >= a.ilo && i <= a.ihi;

    // face geometry
    const bool f_in = ain && iint && ja >= a.jlo - 1 && ja <= a.jhi;
    C QU = C(0), cfl = C(0), ahd = C(0);
    bool up = false, uu_ok = false, act = false;
    if (f_in) {
        const long long q2 = (long long)ja * s + i;
        act = getm_flux_point(a.umask[q2]);
        if (act) {
            const int m_s = ja > 0 ? a.umask[q2 - s] : 0;
            const int m_n = ja + 1 < a.ny_ ? a.umask[q2 + s] : 0;
            const C vv = hx_c<C>(a.u[base + ja * s]);
            const C hvf = hx_c<C>(a.hu[base + ja * s]);
            const C dxf = hx_dy<C>(a)[q2], idyf = hx_idx<C>(a)[q2];
            QU = hx_mul3(vv, hvf, dxf);
            cfl = hx_abs(hx_mul3(vv, hx_dt<C>(a), idyf));
            up = hx_positive(vv);
            uu_ok = getm_flux_point(up ? m_s : m_n);
            if (a.Ah) ahd = hx_ahd(hx_c<C>(a.Ah[q2]), hvf, idyf, dxf);
        }
    }
    sx[ty][tx] = QU;
    __syncthreads();
    const C QUn = ty + 1 < BY ? sx[ty + 1][tx] : C(0);  // north face of cell jb

    const bool bin = ty < (BY - 1) && icol && jb < a.ny_;
    const bool upd = bin && iint && jb >= a.jlo && jb <= a.jhi && a.tmask[(long long)jb * s + i] == 1;
    C coef = C(0);
    double hnew = 0.0;
    if (bin) {
        const double hold = a.h_in[base + jb * s];
        hnew = hold;
        if (upd) hx_cell(hx_dt<C>(a), QUn, QU, hx_iA<C>(a)[(long long)jb * s + i], hold, hnew, coef);
        a.h_out[base + jb * s] = hnew;
    }
    // staging rows: thread row ty loads row ja (smem row ty + 1); rows 0-2
    // also load rows j0-2, j0+BY-1 and j0+BY (smem rows 0, BY+1, BY+2)
    const int jx = ty == 0 ? j0 - 2 : j0 + BY - 2 + ty;
    const int sxrow = ty == 0 ? 0 : BY + ty;
    const bool xin = ty < 3 && icol && jx >= 0 && jx < a.ny_;
    const TvdFace<C> tf = hx_tvd(a.scheme, cfl, QU);
    for (int t = 0; t < a.ntracer; t++) {
        const S* __restrict__ f = a.fin[t] + base;
        __syncthreads();  // previous tracer's reads of sf, sd and sx are done
        sf[ty + 1][tx] = ain ? f[ja * s] : S(0);
        if (ty < 3) sf[sxrow][tx] = xin ? f[jx * s] : S(0);
        __syncthreads();
        // difference across this thread's face (smem row ty + 1 of sd); rows
        // 0 and 1 also form the differences below and above the block's faces
        sd[ty + 1][tx] = hx_c<C>(sf[ty + 2][tx] - sf[ty + 1][tx]);
        if (ty == 0) sd[0][tx] = hx_c<C>(sf[1][tx] - sf[0][tx]);
        if (ty == 1) sd[BY + 1][tx] = hx_c<C>(sf[BY + 2][tx] - sf[BY + 1][tx]);
        __syncthreads();
        const C dprev = sd[ty][tx], d = sd[ty + 1][tx], dnext = sd[ty + 2][tx];
        const S fb = sf[ty + 2][tx];
        C el = C(0), er = C(0);
        if (act) hx_face(tf, up, uu_ok, QU, dprev, d, dnext, ahd, a.Ah != nullptr, el, er);
        sx[ty][tx] = el;
        __syncthreads();
        const C el_n = ty + 1 < BY ? sx[ty + 1][tx] : C(0);
        if (bin) {
            const S fn = upd ? hx_new(fb, coef, el_n, er) : fb;
            a.fout[t][base + jb * s] = fn;
            if (t == 0) epi(base + jb * s, jb, (double)fn, hnew);
        }
    }
}


// y-direction pass in increment form, marching north.  A warp owns 32
// columns of one layer and a chunk of a.ych cells along y.  Walking the
// faces j = j0-1 .. j0+a.ych-1 it keeps the last four rows of every tracer,
// the three differences around the face and the south face's QU and er in
// registers, so each step issues one independent load per field and row
// (no shared memory, no block barriers) and updates cell j from its south
// face (the previous step) and its north face (this step).  The arithmetic
// is that of hpass_y_inc_body, operation for operation; NT tracers are
// marched together, larger batches in groups of NT in warps of their own (the
// face geometry is reloaded per group).

template <typename S, int NT, typename V = S, typename C = float>
__device__ __forceinline__ void hpass_y_march_body(const HPassArgs<S, V>& a, int bx, int chunk, int k, int lane,
                                                   int t0)
{
    const int i = bx * 32 + lane;
    const long long s = a.nx_;
    const bool icol = i < a.nx_;
    const int ic = icol ? i : a.nx_ - 1;  // in-bounds column for the loads of idle lanes
    const long long base = (long long)k * a.plane + ic;
    const bool iint = icol && i >= a.ilo && i <= a.ihi;
    const int jc0 = chunk * a.ych;
    const int jc1 = min(jc0 + a.ych, a.ny_);
    const int nt = min(NT, a.ntracer - t0);
    const bool first_group = t0 == 0;
    // tracers q >= nt of the group (none when ntracer is 0) read as zero
    const S* f[NT];
    S* fo[NT];
#pragma unroll
    for (int q = 0; q < NT; q++) {
        f[q] = q < nt ? a.fin[t0 + q] + base : nullptr;
        fo[q] = q < nt ? a.fout[t0 + q] + base : nullptr;
    }
    auto rowv = [&](const S* p, int j) -> S {
        return (p && j >= 0 && j < a.ny_ && icol) ? p[(long long)j * s] : S(0);
    };
    auto umask_at = [&](int j) -> int { return (j >= 0 && j < a.ny_) ? a.umask[(long long)j * s + ic] : 0; };

    // window at the first face j = jc0 - 1: rows j-1 .. j+1 and d(j-1), d(j)
    S fm1[NT], f0[NT], f1[NT];
    C dm1[NT], d0[NT], er_s[NT];
#pragma unroll
    for (int q = 0; q < NT; q++) {
        fm1[q] = rowv(f[q], jc0 - 2);
        f0[q] = rowv(f[q], jc0 - 1);
        f1[q] = rowv(f[q], jc0);
        dm1[q] = hx_c<C>(f0[q] - fm1[q]);
        d0[q] = hx_c<C>(f1[q] - f0[q]);
        er_s[q] = C(0);
    }
    int m_m = umask_at(jc0 - 2), m_0 = umask_at(jc0 - 1);
    C QU_s = C(0);
    // every load of step j
    struct StepLoads {
        int m_1, tm;
        S f2[NT];
        V uraw;
        double huraw, hold;
        C dxf, idyf, ahraw, iaf;
    };
    auto load_step = [&](int j) -> StepLoads {
        StepLoads L;
        L.m_1 = umask_at(j + 1);
#pragma unroll
        for (int q = 0; q < NT; q++) L.f2[q] = rowv(f[q], j + 2);
        const long long jr = (long long)((j >= 0 && j < a.ny_) ? j : 0) * s;
        L.uraw = a.u[base + jr];
        L.huraw = a.hu[base + jr];
        L.dxf = hx_dy<C>(a)[jr + ic];
        L.idyf = hx_idx<C>(a)[jr + ic];
        L.ahraw = a.Ah ? hx_c<C>(a.Ah[jr + ic]) : C(0);
        L.hold = a.h_in[base + jr];
        L.tm = a.tmask[jr + ic];
        L.iaf = hx_iA<C>(a)[jr + ic];
        return L;
    };
    // one tracer: prefetch a step ahead (more loads in flight per warp);
    // two: the registers go to occupancy instead
    constexpr bool PF = NT == 1;
    StepLoads nxt = load_step(jc0 - 1);
    for (int j = jc0 - 1; j < jc1; j++) {
        const StepLoads cur = PF ? nxt : load_step(j);
        if (PF) nxt = load_step(min(j + 1, jc1 - 1));
        const int m_1 = cur.m_1;
        const S* f2 = cur.f2;
        const bool jin = j >= 0 && j < a.ny_;
        const long long jr = (long long)(jin ? j : 0) * s;
        const V uraw = cur.uraw;
        const double huraw = cur.huraw;
        const C dxf = cur.dxf, idyf = cur.idyf, ahraw = cur.ahraw;
        const double hold = cur.hold;
        const int tm = cur.tm;
        const C iaf = cur.iaf;

        // face j (between cells j and j+1)
        const bool f_in = jin && iint && j >= a.jlo - 1 && j <= a.jhi;
        C QU = C(0), cfl = C(0), ahd = C(0);
        bool up = false, uu_ok = false, act = false;
        if (f_in) {
            act = getm_flux_point(m_0);
            if (act) {
                const C vv = hx_c<C>(uraw);
                const C hvf = hx_c<C>(huraw);
                QU = hx_mul3(vv, hvf, dxf);
                cfl = hx_abs(hx_mul3(vv, hx_dt<C>(a), idyf));
                up = hx_positive(vv);
                uu_ok = getm_flux_point(up ? m_m : m_1);
                if (a.Ah) ahd = hx_ahd(ahraw, hvf, idyf, dxf);
            }
        }
        // cell j: south face j-1 (previous step), north face j (this step)
        const bool upd_cell = j >= jc0 && iint && j >= a.jlo && j <= a.jhi && tm == 1;
        C coef = C(0);
        double hnew = hold;
        if (upd_cell) hx_cell(hx_dt<C>(a), QU, QU_s, iaf, hold, hnew, coef);
        if (j >= jc0 && icol && first_group) a.h_out[base + jr] = hnew;
        const TvdFace<C> tf = hx_tvd(a.scheme, cfl, QU);
#pragma unroll
        for (int q = 0; q < NT; q++) {
            const C d1 = hx_c<C>(f2[q] - f1[q]);
            C el = C(0), er = C(0);
            if (act)
                hx_face(tf, up, uu_ok, QU, dm1[q], d0[q], d1, ahd, a.Ah != nullptr, el, er);
            if (j >= jc0 && icol && q < nt) fo[q][jr] = upd_cell ? hx_new(f0[q], coef, el, er_s[q]) : f0[q];
            er_s[q] = er;
            fm1[q] = f0[q]; f0[q] = f1[q]; f1[q] = f2[q];
            dm1[q] = d0[q]; d0[q] = d1;
        }
        QU_s = QU;
        m_m = m_0; m_0 = m_1;
    }
}

// ---------------------------------------------------------------------------
// The two passes of a FULL-split 2D advection (advection_2d_impl with split
// 1, no horizontal diffusion), set up for kernels that run them themselves:
// first: var -> scratch, D -> scratch thickness; second: back into var and
// D.  Implemented in advection.cu (it owns the scratch buffers).
// ---------------------------------------------------------------------------
struct Advection2DPasses {
    HPassArgs<double> pass[2];
    int dir[2];  // 1: x pass, 2: y pass
};

int getm_advection_2d_passes(getm_advection* adv, getm_grid* tgrid, getm_grid* ugrid, getm_grid* vgrid,
                             int ufirst, const double* u, const double* v, double timestep, double* D,
                             const double* DU, const double* DV, double* var, int increment,
                             Advection2DPasses* out);
