// Implicit (Crank-Nicolson) vertical diffusion for sm_103a.
//
// Reference: src/operators/diffusion.F90 (prepare :135-204, apply :206-314)
// reached through python/src/wrapper.F90:127-186 and
// python/pygetm/operators.py:218-230 (VerticalDiffusion).
//
// GB300 design: one thread per water column.  The C layout [k][j][i] puts the
// 32 columns of a warp next to each other at every level, so each per-level
// load/store of the sweep is a fully coalesced 256-byte transaction.  The
// tridiagonal matrix is never stored: its coefficients are formed on the fly
// from nuh, ho, hn and var while sweeping down from the surface (the Thomas
// forward elimination of diffusion.F90:285-292), keeping only the two
// coefficients per level for the back substitution (:304-307), in shared
// memory or in a caller-provided global workspace.  prepare+apply are fused
// (traffic per field: read nuh, ho, hn, var [+ea2, ea4], write var).  The mixed form's solve (vd_inc_kernel) takes fields in pairs and
// issues each level's loads one level ahead.  A warp-per-column PCR solve would
// cost O(nz log nz) FP64 divides per column instead of O(nz); GB300's FP64
// rate makes the serial Thomas sweep the faster choice for the FP64 form.
// For domains with few columns the mixed form can instead split each column
// into four segments, one warp each (vd_seg_kernel, the partition method).
#include <stdlib.h>
#include <string.h>

#include "getm_common.cuh"

#define VD_MAX_BATCH 32

struct getm_vertical_diffusion {
    getm_grid* tgrid;
    size_t n3;
    double* auxo;   // prepare -> apply work arrays (diffusion.F90:88)
    double* auxn;
};

// T: type of nuh and of the solve (double: FP64 form; float: mixed form);
// S: storage type of the diffused fields (T unless given; double with a
// float solve: the mixed form with FP64 tracer storage, increment form).
// Layer thicknesses are double in every form.
template <typename T, typename S = T>
struct VDArgs {
    int nx_, ny_, nz;
    long long plane;
    const int* mask;
    const T* nuh;          // nz+1 interface levels
    const double* ho;
    const double* hn;
    const double* auxo;    // FP64 form, when prepared separately (else NULL)
    const double* auxn;
    double dt, cnpar;
    int ntracer;
    double molecular[VD_MAX_BATCH];
    S* var[VD_MAX_BATCH];
    const T* ea2[VD_MAX_BATCH];
    const T* ea4[VD_MAX_BATCH];
    T* work;               // NULL, or 2 nz plane elements: elimination coefficients in global memory
};

// A layer thickness in the solve's type (the mixed form converts on the
// integer pipe, see getm_d2f_approx).
template <typename T>
__device__ __forceinline__ T vd_h(double h)
{
    if constexpr (getm_increment_form<T>) return getm_d2f_approx(h);
    else return h;
}

// Coupling coefficients of the interface above C level k (between levels k and
// k+1): diffusion.F90:166-168 with Fortran k = C k + 1.
__device__ __forceinline__ void vd_aux(const VDArgs<float>& a, long long c, int k, double mol, float& auxo,
                                       float& auxn)
{
    const long long P = a.plane;
    float x = (float)(2.0 * a.dt) * (a.nuh[c + (k + 1) * P] + (float)mol);
    auxo = (float)(1.0 - a.cnpar) * x / (vd_h<float>(a.ho[c + (k + 1) * P]) + vd_h<float>(a.ho[c + k * P]));
    auxn = (float)a.cnpar * x / (vd_h<float>(a.hn[c + (k + 1) * P]) + vd_h<float>(a.hn[c + k * P]));
}

// Increment form: (ho - hn) of one layer as float, exact-difference first;
// zero without FP64 work when the solve uses one thickness (ho == hn).
__device__ __forceinline__ float vd_dh(const double* ho, const double* hn, long long q)
{
    return ho == hn ? 0.f : getm_d2f_approx(ho[q] - hn[q]);
}

// A single layer (diffusion.F90:224-231): every point, mask not consulted.
template <typename T, typename S>
__device__ __forceinline__ void vd_single_layer(const VDArgs<T, S>& a, long long c)
{
    for (int t = 0; t < a.ntracer; t++) {
        const S x = a.var[t][c];
        T a2 = vd_h<T>(a.hn[c]);
        if constexpr (getm_increment_form<T>) {
            const float xf = inc_f<S>(x);
            float r = xf * vd_dh(a.ho, a.hn, c);
            if (a.ea2[t]) { a2 = a2 - a.ea2[t][c]; r = r + a.ea2[t][c] * xf; }
            if (a.ea4[t]) r = r + a.ea4[t][c];
            a.var[t][c] = inc_add<S>(x, r / a2);
        } else {
            if (a.ea2[t]) a2 = a2 - a.ea2[t][c];
            T a4 = a.ho[c] * x;
            if (a.ea4[t]) a4 = a4 + a.ea4[t][c];
            a.var[t][c] = a4 / a2;
        }
    }
}

// The solves work in increments: with x the old values and A x_new = a4 the
// reference system, they solve A dx = a4 - A x, whose right-hand side reduces
// to differences of neighbouring values
//   r_k = x_k (ho_k - hn_k) + (x_{k+1} - x_k)(auxo + auxn)_{k+1/2}
//         + (x_{k-1} - x_k)(auxo + auxn)_{k-1/2} + ea4_k + ea2_k x_k
// and write x + dx, so rounding scales with the change of the field.
//
// FP64 form, thread per column.  GB300's FP64 rate bounds it, so it counts
// FP64 instructions: one reciprocal per row and per interface (getm_rcp) in
// place of the reference's four divisions and none for the explicit half of
// the coupling when cnpar = 1: 20 per level, where the reference's order of
// evaluation took about 130.  Eliminating downwards from the surface, with up
// and lo the implicit couplings above and below a row, F = (auxo + auxn) (x_{k-1}
// - x_k) the old field's flux term and src the remaining terms of r_k,
//     t = hn - ea2 + up s',  den = t + lo,  r = lo / den,  s = t / den,
//     y = s F + r (y' - src),
// where ' marks the row above (zero at the surface), and upwards
//     dx_k = r (x_{k-1} - x_k + dx_{k-1}) + (src + auxo (x_{k-1} - x_k) - y') / den.
// Here t is the row's diagonal less lo (1 + the reference's r_k is s) and y the
// flux left over from the rows above: no large terms are subtracted, so strong
// mixing costs no digits (the reference's a2 - a3 r_k loses about lo / hn ulps).
// As in vd_inc_sweep every operand of a level is loaded one level ahead.
// Measured: 120 x 100 x 30, one field, 103 -> 41 us; 200 x 150 x 30, two fields with
// sources and two thicknesses, 286 -> 130 us; error against quad precision
// 1.3e-16 -> 0.5e-16.
// r and the second term of dx are kept at stride rs per level, in shared
// memory or the caller's workspace ([k][j][i]).  Prepared coupling
// coefficients (a.auxo) replace those formed here.
template <bool SRC>
__device__ __forceinline__ void vd_f64_sweep(const VDArgs<double>& a, long long c, int t, double* ru, double* qu,
                                             long long rs)
{
    const long long P = a.plane;
    const int nz = a.nz;
    const double* __restrict__ ho = a.ho + c;
    const double* __restrict__ hn = a.hn + c;
    const bool one_h = a.ho == a.hn, prep = a.auxo != nullptr;
    const bool both = prep || a.cnpar != 1.0;  // an explicit half too
    const bool use_ho = !one_h;
    const double dt2 = 2.0 * a.dt, co = 1.0 - a.cnpar, mol = a.molecular[t];
    double* v = a.var[t] + c;
    const double* e2 = SRC && a.ea2[t] ? a.ea2[t] + c : nullptr;
    const double* e4 = SRC && a.ea4[t] ? a.ea4[t] + c : nullptr;
    // level k operands (current) and the raw loads of level k-1 (next)
    int k = nz - 1;
    double ho_c = use_ho ? ho[k * P] : 0.0, ho_n = use_ho ? ho[(k - 1) * P] : 0.0;
    double hn_c = hn[k * P], hn_n = hn[(k - 1) * P];
    double nuh_c = prep ? 0.0 : a.nuh[c + k * P];  // interface below level k
    double vk = v[k * P], vn = v[(k - 1) * P];
    double e2c = SRC && e2 ? e2[k * P] : 0.0, e4c = SRC && e4 ? e4[k * P] : 0.0;
    double up = 0.0, sp = 0.0, yp = 0.0;  // of the row above
    double dx = 0.0;
    for (; k >= 0; k--) {
        // the raw operands of level k-2 and of the interface below level k-1
        double ho_nn = 0.0, hn_nn = 0.0, nuh_n = 0.0, vnn = 0.0, e2n = 0.0, e4n = 0.0;
        if (k >= 2) {
            if (use_ho) ho_nn = ho[(k - 2) * P];
            hn_nn = hn[(k - 2) * P];
            vnn = v[(k - 2) * P];
        }
        if (k >= 1) {
            if (!prep) nuh_n = a.nuh[c + (k - 1) * P];
            if (SRC && e2) e2n = e2[(k - 1) * P];
            if (SRC && e4) e4n = e4[(k - 1) * P];
        }
        // y' - src of this row, and t
        double hk = hn_c, ys = yp;
        if (use_ho) ys = __fma_rn(-vk, __dadd_rn(ho_c, -hn_c), ys);
        if (SRC && e2) {
            hk = __dadd_rn(hk, -e2c);
            ys = __fma_rn(-e2c, vk, ys);
        }
        if (SRC && e4) ys = __dadd_rn(ys, -e4c);
        const double tk = __fma_rn(up, sp, hk);
        if (k == 0) {  // no interface below
            dx = -__dmul_rn(ys, getm_rcp(tk));
            break;
        }
        // the interface below level k: lo implicit, eo explicit
        double lo, eo = 0.0;
        if (prep) {
            lo = a.auxn[c + (k - 1) * P];
            eo = a.auxo[c + (k - 1) * P];
        } else {
            const double x = __dmul_rn(dt2, __dadd_rn(nuh_c, mol));
            const double rsn = getm_rcp(__dadd_rn(hn_c, hn_n));
            if (both) {
                lo = __dmul_rn(__dmul_rn(a.cnpar, x), rsn);
                eo = __dmul_rn(__dmul_rn(co, x), one_h ? rsn : getm_rcp(__dadd_rn(ho_c, ho_n)));
            } else {
                lo = __dmul_rn(x, rsn);
            }
        }
        const double dd = __dadd_rn(vn, -vk);
        const double inv = getm_rcp(__dadd_rn(tk, lo));
        const double r = __dmul_rn(lo, inv);
        // s F = (t / den) lo dd = r t dd, and the explicit half's part
        double q = ys;
        sp = __dmul_rn(tk, inv);
        yp = __dmul_rn(r, __fma_rn(tk, dd, ys));
        if (both) {
            const double fe = __dmul_rn(eo, dd);
            yp = __fma_rn(sp, fe, yp);
            q = __dadd_rn(q, -fe);
        }
        ru[k * rs] = r;
        qu[k * rs] = -__dmul_rn(q, inv);
        up = lo;
        vk = vn; vn = vnn;
        e2c = e2n; e4c = e4n;
        hn_c = hn_n; hn_n = hn_nn;
        ho_c = ho_n; ho_n = ho_nn;
        nuh_c = nuh_n;
    }
    // back substitution (:304-307)
    double xn = v[P], rn = ru[rs], qn = qu[rs];
    double below = __dadd_rn(vk, dx);  // the new value of the level below
    v[0] = below;
    for (k = 1; k < nz; k++) {
        const double x_old = xn, r = rn, q = qn;
        if (k + 1 < nz) {
            xn = v[(k + 1) * P];
            rn = ru[(k + 1) * rs];
            qn = qu[(k + 1) * rs];
        }
        below = __dadd_rn(x_old, __fma_rn(r, __dadd_rn(below, -x_old), q));
        v[k * P] = below;
    }
}

// Blocks of 32 columns by blockDim.y rows, one field after the other (the
// workspace a caller brings holds one field's coefficients: 2 nz planes, or NULL
// for shared memory), or side by side in blocks z.
template <bool SRC>
__global__ void __launch_bounds__(128, 5) vd_f64_kernel(VDArgs<double> a)
{
    extern __shared__ __align__(16) unsigned char vd_smem[];
    const int i = blockIdx.x * 32 + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    if (i >= a.nx_ || j >= a.ny_) return;
    const long long c = (long long)j * a.nx_ + i;
    if (a.nz == 1) {
        vd_single_layer(a, c);
        return;
    }
    if (a.mask[c] != 1) return;
    double* const ru = a.work ? a.work + c : (double*)vd_smem + threadIdx.y * 32 + threadIdx.x;
    const long long rs = a.work ? a.plane : 32 * (long long)blockDim.y;
    for (int t = blockIdx.z; t < a.ntracer; t += gridDim.z) vd_f64_sweep<SRC>(a, c, t, ru, ru + a.nz * rs, rs);
}

// Float solve without a workspace, thread per column; dynamic shared memory
// holds ru, qu and the old values: 3 nz blockDim values.
constexpr int VD_SMEM_ARRAYS = 3;

__global__ void __launch_bounds__(128, 8) vd_column_kernel(VDArgs<float> a)
{
    extern __shared__ __align__(16) unsigned char vd_smem[];
    const int tid = threadIdx.x;
    const int nthreads = blockDim.x;
    const int i = blockIdx.x * blockDim.x + tid;
    const int j = blockIdx.y;
    if (i >= a.nx_) return;
    const long long c = (long long)j * a.nx_ + i;
    const long long P = a.plane;
    const int nz = a.nz;
    if (nz == 1) {
        vd_single_layer(a, c);
        return;
    }
    if (a.mask[c] != 1) return;
    float* ru = (float*)vd_smem + tid;
    float* qu = ru + (size_t)nz * nthreads;
    float* xo = qu + (size_t)nz * nthreads;
    const int rs = nthreads;
    for (int t = 0; t < a.ntracer; t++) {
        float* __restrict__ var = a.var[t];
        const float* ea2 = a.ea2[t];
        const float* ea4 = a.ea4[t];
        const double mol = a.molecular[t];
        // surface layer (C level nz-1), diffusion.F90:238-245
        int k = nz - 1;
        float aob, anb;                         // aux of the interface below level k
        vd_aux(a, c, k - 1, mol, aob, anb);
        float vk = var[c + k * P];
        float vkm1 = var[c + (k - 1) * P];
        float a1 = -anb;
        float a2 = vd_h<float>(a.hn[c + k * P]) + anb;
        xo[k * rs] = vk;
        float a4 = vk * vd_dh(a.ho, a.hn, c + k * P) + (vkm1 - vk) * (aob + anb);
        if (ea2) a4 = a4 + ea2[c + k * P] * vk;
        if (ea2) a2 = a2 - ea2[c + k * P];
        if (ea4) a4 = a4 + ea4[c + k * P];
        float rk = a1 / a2;
        float qk = a4 / a2;
        ru[k * rs] = rk;
        qu[k * rs] = qk;
        // inner layers, diffusion.F90:247-258 and elimination :287-290
        float aoa = aob, ana = anb;             // interface above level k-1
        float vkp1 = vk;
        vk = vkm1;
        for (k = nz - 2; k >= 1; k--) {
            vd_aux(a, c, k - 1, mol, aob, anb);
            vkm1 = var[c + (k - 1) * P];
            float a3 = -ana;
            a1 = -anb;
            a2 = vd_h<float>(a.hn[c + k * P]) + ana + anb;
            xo[k * rs] = vk;
            a4 = vk * vd_dh(a.ho, a.hn, c + k * P) + (vkp1 - vk) * (aoa + ana) + (vkm1 - vk) * (aob + anb);
            if (ea2) a4 = a4 + ea2[c + k * P] * vk;
            if (ea2) a2 = a2 - ea2[c + k * P];
            if (ea4) a4 = a4 + ea4[c + k * P];
            float den = a2 - a3 * rk;
            rk = a1 / den;
            qk = (a4 - a3 * qk) / den;
            ru[k * rs] = rk;
            qu[k * rs] = qk;
            aoa = aob; ana = anb;
            vkp1 = vk; vk = vkm1;
        }
        // bottom layer, diffusion.F90:260-267 and :291-292
        float a3 = -ana;
        a2 = vd_h<float>(a.hn[c]) + ana;
        a4 = vk * vd_dh(a.ho, a.hn, c) + (vkp1 - vk) * (aoa + ana);
        if (ea2) a4 = a4 + ea2[c] * vk;
        if (ea2) a2 = a2 - ea2[c];
        if (ea4) a4 = a4 + ea4[c];
        float vprev = (a4 - a3 * qk) / (a2 - a3 * rk);
        // back substitution :304-307
        var[c] = vk + vprev;
        for (k = 1; k < nz; k++) {
            vprev = qu[k * rs] - ru[k * rs] * vprev;
            var[c + k * P] = xo[k * rs] + vprev;
        }
    }
}

// Increment form of the float solve with the elimination coefficients in global
// or shared memory: the arithmetic of vd_column_kernel, restructured for
// memory-level parallelism.  The loads of the
// forward elimination do not depend on the elimination itself, so the
// operands of the next level (thicknesses, nuh, field values, sources) are
// issued one level ahead of the arithmetic, and those of the back
// substitution likewise; NT fields share the thickness and nuh loads and
// sweep together (work: 2 nz planes per field of a group).  SRC: whether a
// field of the group has ea2 or ea4 (without, no registers are spent on
// them).
// coef, rs: the thread's coefficients of the surface level and their stride.
// Pairs (domains of many columns) also ask for the operands of
// the level VD_AHEAD levels further into the cache: their streams come from
// DRAM, and one level ahead does not cover that (400 x 300 x 40, two FP64-stored
// fields, 134 -> 118 us; where one field sweeps alone the extra instructions
// cost 5 %, and two float fields with sources gain nothing).
constexpr int VD_AHEAD = 3;

template <typename T>
__device__ __forceinline__ void vd_prefetch(const T* p)
{
    asm volatile("prefetch.global.L1 [%0];" ::"l"(p));
}

template <int NT, bool SRC, typename S>
__device__ __forceinline__ void vd_inc_sweep(const VDArgs<float, S>& a, long long c, int t0, float* coef, long long rs)
{
    const long long P = a.plane;
    const int nz = a.nz;
    const double* __restrict__ ho = a.ho + c;
    const double* __restrict__ hn = a.hn + c;
    const float* __restrict__ nuh = a.nuh + c;
    const bool one_h = a.ho == a.hn;
    const float co = (float)(1.0 - a.cnpar), cn = (float)a.cnpar, dt2 = (float)(2.0 * a.dt);
    S* v[NT];
    const float* e2[NT];
    const float* e4[NT];
    float* ru[NT];
    float* qu[NT];
    float mol[NT];
#pragma unroll
    for (int t = 0; t < NT; t++) {
        v[t] = a.var[t0 + t] + c;
        e2[t] = SRC && a.ea2[t0 + t] ? a.ea2[t0 + t] + c : nullptr;
        e4[t] = SRC && a.ea4[t0 + t] ? a.ea4[t0 + t] + c : nullptr;
        ru[t] = coef + (long long)(2 * t) * nz * rs;
        qu[t] = ru[t] + (long long)nz * rs;
        mol[t] = (float)a.molecular[t0 + t];
    }
    // level k operands (current) and the raw loads of level k-1 (next)
    int k = nz - 1;
    double ho_c = ho[k * P], hn_c = hn[k * P];
    double ho_n = ho[(k - 1) * P], hn_n = hn[(k - 1) * P];
    float nuh_c = nuh[k * P];  // interface below level k
    S vk[NT], vn[NT];
    float e2c[NT], e4c[NT];
#pragma unroll
    for (int t = 0; t < NT; t++) {
        vk[t] = v[t][k * P];
        vn[t] = v[t][(k - 1) * P];
        e2c[t] = SRC && e2[t] ? e2[t][k * P] : 0.f;
        e4c[t] = SRC && e4[t] ? e4[t][k * P] : 0.f;
    }
    float hoF = vd_h<float>(ho_c), hnF = vd_h<float>(hn_c);
    float dh = one_h ? 0.f : getm_d2f_approx(ho_c - hn_c);
    float rk[NT], qk[NT], aoa[NT], ana[NT], dprev[NT];
    // surface layer (diffusion.F90:238-245) and the inner layers
    // (:247-258, elimination :287-290)
    for (; k >= 1; k--) {
        // next level's raw operands, one level ahead
        const int kn = k - 1;
        double ho_nn = 0.0, hn_nn = 0.0;
        float nuh_n = 0.f, e2n[NT], e4n[NT];
        S vnn[NT];
        if (NT > 1 && kn >= 1 + VD_AHEAD) {
            const int kp = kn - 1 - VD_AHEAD;
            vd_prefetch(ho + kp * P);
            if (!one_h) vd_prefetch(hn + kp * P);
            vd_prefetch(nuh + (kp + 1) * P);
#pragma unroll
            for (int t = 0; t < NT; t++) {
                vd_prefetch(v[t] + kp * P);
                if (SRC && e2[t]) vd_prefetch(e2[t] + (kp + 1) * P);
                if (SRC && e4[t]) vd_prefetch(e4[t] + (kp + 1) * P);
            }
        }
        if (kn >= 1) {
            ho_nn = ho[(kn - 1) * P];
            hn_nn = hn[(kn - 1) * P];
        }
        nuh_n = nuh[kn * P];
#pragma unroll
        for (int t = 0; t < NT; t++) {
            vnn[t] = kn >= 1 ? v[t][(kn - 1) * P] : S(0);
            e2n[t] = SRC && e2[t] ? e2[t][kn * P] : 0.f;
            e4n[t] = SRC && e4[t] ? e4[t][kn * P] : 0.f;
        }
        // interface below level k (vd_aux with C level k-1)
        const float hoFn = vd_h<float>(ho_n), hnFn = vd_h<float>(hn_n);
        const float so = hoF + hoFn, sn = hnF + hnFn;
#pragma unroll
        for (int t = 0; t < NT; t++) {
            const float x = dt2 * (nuh_c + mol[t]);
            const float aob = co * x / so;
            const float anb = cn * x / sn;
            const float a1 = -anb;
            // differences of neighbouring values in the storage type, then
            // narrowed (exact for float storage); the difference to the
            // level above is minus the level above's difference to this one
            const float xk = inc_f<S>(vk[t]);
            const float ddn = inc_f<S>(vn[t] - vk[t]);
            float a2, a4;
            if (k == nz - 1) {
                a2 = hnF + anb;
                a4 = xk * dh + ddn * (aob + anb);
            } else {
                a2 = hnF + ana[t] + anb;
                a4 = xk * dh + (-dprev[t]) * (aoa[t] + ana[t]) + ddn * (aob + anb);
            }
            dprev[t] = ddn;
            if (SRC && e2[t]) a4 = a4 + e2c[t] * xk;
            if (SRC && e2[t]) a2 = a2 - e2c[t];
            if (SRC && e4[t]) a4 = a4 + e4c[t];
            if (k == nz - 1) {
                rk[t] = a1 / a2;
                qk[t] = a4 / a2;
            } else {
                const float a3 = -ana[t];
                const float den = a2 - a3 * rk[t];
                rk[t] = a1 / den;
                qk[t] = (a4 - a3 * qk[t]) / den;
            }
            ru[t][k * rs] = rk[t];
            qu[t][k * rs] = qk[t];
            aoa[t] = aob; ana[t] = anb;
            vk[t] = vn[t]; vn[t] = vnn[t];
            e2c[t] = e2n[t]; e4c[t] = e4n[t];
        }
        hoF = hoFn; hnF = hnFn;
        dh = one_h ? 0.f : getm_d2f_approx(ho_n - hn_n);
        ho_n = ho_nn; hn_n = hn_nn;
        nuh_c = nuh_n;
    }
    // bottom layer (:260-267, :291-292), back substitution (:304-307);
    // the old values of level k+1 are read before level k is written
    float vprev[NT], rn[NT], qn[NT];
    S xn[NT];
#pragma unroll
    for (int t = 0; t < NT; t++) {
        const float a3 = -ana[t];
        const float xk = inc_f<S>(vk[t]);
        float a2 = hnF + ana[t];
        float a4 = xk * dh + (-dprev[t]) * (aoa[t] + ana[t]);
        if (SRC && e2[t]) a4 = a4 + e2c[t] * xk;
        if (SRC && e2[t]) a2 = a2 - e2c[t];
        if (SRC && e4[t]) a4 = a4 + e4c[t];
        vprev[t] = (a4 - a3 * qk[t]) / (a2 - a3 * rk[t]);
        xn[t] = v[t][P];
        rn[t] = ru[t][rs];
        qn[t] = qu[t][rs];
        v[t][0] = inc_add<S>(vk[t], vprev[t]);
    }
    for (k = 1; k < nz; k++) {
#pragma unroll
        for (int t = 0; t < NT; t++) {
            const S x_old = xn[t];
            const float r = rn[t], q = qn[t];
            if (NT > 1 && k + 1 + VD_AHEAD < nz) vd_prefetch(v[t] + (k + 1 + VD_AHEAD) * P);
            if (k + 1 < nz) {
                xn[t] = v[t][(k + 1) * P];
                rn[t] = ru[t][(k + 1) * rs];
                qn[t] = qu[t][(k + 1) * rs];
            }
            vprev[t] = q - r * vprev[t];
            v[t][k * P] = inc_add<S>(x_old, vprev[t]);
        }
    }
}

// PAIRS: fields in pairs (then an odd last one alone), else one at a time.
// Blocks of 32 columns by GETM_TUNE_COLUMN_ROWS rows.  S: storage type of
// the fields (float, or double for FP64 tracer storage).  SM (and not
// PAIRS): the coefficients in shared memory and each field in blocks of its own
// (grid z); else in the global workspace, pairs one after the other, or single
// fields in as many blocks (grid z) as the workspace holds fields.
template <bool SRC, bool PAIRS, bool SM, typename S>
__global__ void __launch_bounds__(128, 7) vd_inc_kernel(VDArgs<float, S> a)
{
    extern __shared__ __align__(16) unsigned char vd_smem[];
    const int i = blockIdx.x * 32 + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    if (i >= a.nx_ || j >= a.ny_) return;
    const long long c = (long long)j * a.nx_ + i;
    if (a.nz == 1) {
        if (blockIdx.z == 0) vd_single_layer(a, c);
        return;
    }
    if (a.mask[c] != 1) return;
    if constexpr (SM) {
        float* coef = reinterpret_cast<float*>(vd_smem) + threadIdx.y * 32 + threadIdx.x;
        vd_inc_sweep<1, SRC, S>(a, c, blockIdx.z, coef, 32 * blockDim.y);
    } else {
        int t0 = blockIdx.z;
        if constexpr (PAIRS)
            for (; t0 + 2 <= a.ntracer; t0 += 2) vd_inc_sweep<2, SRC, S>(a, c, t0, a.work + c, a.plane);
        float* coef = a.work + c + (long long)blockIdx.z * 2 * a.nz * a.plane;
        for (; t0 < a.ntracer; t0 += gridDim.z) vd_inc_sweep<1, SRC, S>(a, c, t0, coef, a.plane);
    }
}

// Whether the fields of a batch may be swept side by side: none lies in memory
// that the sweep of another one reads or writes (a field given twice, or as
// another's source: those are swept in turn).
template <typename T, typename S>
static bool vd_fields_apart(const VDArgs<T, S>& a)
{
    const size_t n = (size_t)a.plane * a.nz;
    for (int t = 0; t < a.ntracer; t++) {
        const char* const f = (const char*)a.var[t];
        auto apart = [&](const void* q, size_t bytes) {
            return !q || f + n * sizeof(S) <= (const char*)q || (const char*)q + bytes <= f;
        };
        if (!apart(a.nuh, (n + a.plane) * sizeof(T)) || !apart(a.ho, n * sizeof(double)) || !apart(a.hn, n * sizeof(double)))
            return false;
        for (int s = 0; s < a.ntracer; s++)
            if (s != t && !(apart(a.var[s], n * sizeof(S)) && apart(a.ea2[s], n * sizeof(T)) && apart(a.ea4[s], n * sizeof(T))))
                return false;
    }
    return true;
}

template <bool SRC, typename S>
static int vd_inc_launch_src(VDArgs<float, S>& a, cudaStream_t stream)
{
    const int rows = getm_tune(GETM_TUNE_COLUMN_ROWS);
    dim3 grid(getm_div_up(a.nx_, 32), getm_div_up(a.ny_, rows)), block(32, rows);
    // Several fields on a domain with few columns (a sweep is then a chain of
    // latencies): each field in blocks of its own, up to 20 warps of columns per
    // SM, and up to the layers whose coefficients leave room for 20 warps per
    // SM.  us, pairs in turn through the workspace -> fields side by side: 92 x 92
    // x 20 two fields 31 -> 21; 150 x 120 x 30 three 80 -> 35; 240 x 200 x 20
    // eight 155 -> 79 (pairs side by side 118); 300 x 250 x 25 two 60 -> 52; but
    // 400 x 300 x 40 two (26 warps) 133 -> 164, and one field alone 75 -> 103.
    const long long warps = (long long)grid.x * a.ny_;
    const bool side = a.ntracer > 1 && warps <= 20 * GETM_SMS && vd_fields_apart(a);
    if (side && a.nz <= 45) {
        const size_t smem = (size_t)rows * 32 * a.nz * 2 * sizeof(float);  // at most 45 KB
        static std::atomic<unsigned long long> done{0};
        if (!getm_once_per_device(done, [] {
                return cudaFuncSetAttribute(vd_inc_kernel<SRC, false, true, S>,
                                            cudaFuncAttributePreferredSharedMemoryCarveout, 100) == cudaSuccess;
            }))
            return GETM_ERR_CUDA;
        grid.z = a.ntracer;
        vd_inc_kernel<SRC, false, true, S><<<grid, block, smem, stream>>>(a);
    } else if (side && warps <= 10 * GETM_SMS) {
        // more layers, up to ten warps per SM: through the workspace, which holds two
        // fields' coefficients.  us, pairs in turn -> these: 64 x 48 x 60 two
        // float fields 81 -> 50, with sources 105 -> 52, FP64-stored 96 -> 57; 200 x
        // 150 x 60 FP64-stored 108 -> 80
        grid.z = 2;
        vd_inc_kernel<SRC, false, false, S><<<grid, block, 0, stream>>>(a);
    } else if (a.ntracer > 1) {
        vd_inc_kernel<SRC, true, false, S><<<grid, block, 0, stream>>>(a);
    } else {
        vd_inc_kernel<SRC, false, false, S><<<grid, block, 0, stream>>>(a);
    }
    GETM_CHECK_LAUNCH();
    return GETM_OK;
}

template <typename S>
static int vd_inc_launch(VDArgs<float, S>& a, cudaStream_t stream)
{
    bool src = false;
    for (int t = 0; t < a.ntracer; t++) src = src || a.ea2[t] || a.ea4[t];
    return src ? vd_inc_launch_src<true, S>(a, stream) : vd_inc_launch_src<false, S>(a, stream);
}

// ---------------------------------------------------------------------------
// Segmented column solve (mixed form): VD_NSEG warps share 32 columns
// ---------------------------------------------------------------------------
// The partition method for tridiagonal systems (H. H. Wang, ACM Trans. Math.
// Softw. 7 (1981) 170-183), in the thread-per-segment form of the hybrid
// Thomas/PCR solvers (A. Laszlo, M. Giles, J. Appleyard, ACM Trans. Math.
// Softw. 42 (2016) 31).  Warp s of a block owns levels klo..khi (about
// nz / VD_NSEG of them) of the block's 32 columns; lane i is column i, so
// every load and store is still a coalesced 128- or 256-byte row of a level.
// Each thread
//   1. forms the rows of its levels with the arithmetic of vd_inc_sweep
//      (the increment form: A dx = a4 - A x) and, sweeping up, eliminates
//      each row's coupling to the level below in favour of the segment's
//      first unknown, then, sweeping down through shared memory, the
//      coupling to the level above in favour of its last unknown, so that
//      dx_i = d_i - a_i dx_first - g_i dx_last inside the segment;
//   2. adds the rows of its first and last unknown to a reduced tridiagonal
//      system of 2 VD_NSEG unknowns per column, which warp 0 solves by
//      Thomas elimination in shared memory;
//   3. substitutes the two back into its levels and adds the increments to
//      the stored values.
// A column's chain of dependent steps is VD_NSEG times shorter than the
// serial sweep's, and the elimination coefficients stay in shared memory
// (no global workspace).  It costs one reciprocal and about twice the
// multiply-adds per row and level; the rounding differs from the serial
// sweep's by float rounding of the increments.  Used for 2 VD_NSEG <= nz <=
// VD_NSEG * VD_SEG_MAXM when the GETM_TUNE_COLUMN_SOLVE knob asks for it.
constexpr int VD_NSEG = 4;
constexpr int VD_SEG_MAXM = 16;
constexpr int VD_SEG_THREADS = 32 * VD_NSEG;

// Shared memory of one launch: 3 NT (maxm - 2) per-level coefficients per
// thread (levels strictly inside a segment), and the reduced systems of the
// block's 32 columns (lower, diagonal, upper, right-hand side; the solution
// overwrites the right-hand side).
static size_t vd_seg_smem(int nz, int nt)
{
    const int maxm = (nz + VD_NSEG - 1) / VD_NSEG;
    return sizeof(float) * ((size_t)3 * nt * (maxm > 2 ? maxm - 2 : 0) * VD_SEG_THREADS +
                            (size_t)4 * nt * 2 * VD_NSEG * 32);
}

template <int NT, bool SRC, typename S>
__device__ __forceinline__ void vd_seg_group(const VDArgs<float, S>& a, long long c, bool act, int t0, int s,
                                             int klo, int m, int slots, float* __restrict__ rows,
                                             float* __restrict__ red, int tid, int tx)
{
    constexpr int R = 2 * VD_NSEG;
    const long long P = a.plane;
    const int nz = a.nz;
    // coefficient q (0: a, 1: g, 2: d) of field t at inner level ii (1..m-2)
#define VD_ROW(t, q, ii) rows[(((t) * 3 + (q)) * slots + (ii) - 1) * VD_SEG_THREADS + tid]
    // reduced system of this column: q 0 lower, 1 diagonal, 2 upper, 3 rhs
#define VD_RED(t, q, r) red[(((t) * 4 + (q)) * R + (r)) * 32 + tx]
    if (act) {
        const double* __restrict__ ho = a.ho + c;
        const double* __restrict__ hn = a.hn + c;
        const float* __restrict__ nuh = a.nuh + c;
        const bool one_h = a.ho == a.hn;
        const float co = (float)(1.0 - a.cnpar), cn = (float)a.cnpar, dt2 = (float)(2.0 * a.dt);
        S* v[NT];
        const float* e2[NT];
        const float* e4[NT];
        float mol[NT];
#pragma unroll
        for (int t = 0; t < NT; t++) {
            v[t] = a.var[t0 + t] + c;
            e2[t] = SRC && a.ea2[t0 + t] ? a.ea2[t0 + t] + c : nullptr;
            e4[t] = SRC && a.ea4[t0 + t] ? a.ea4[t0 + t] + c : nullptr;
            mol[t] = (float)a.molecular[t0 + t];
        }
        // level k = klo; the interface below it (k >= 1)
        int k = klo;
        float hoF = vd_h<float>(ho[k * P]), hnF = vd_h<float>(hn[k * P]);
        float dh = one_h ? 0.f : getm_d2f_approx(ho[k * P] - hn[k * P]);
        S xc[NT];
        float aob[NT], anb[NT], ddn[NT];
#pragma unroll
        for (int t = 0; t < NT; t++) {
            xc[t] = v[t][k * P];
            aob[t] = anb[t] = ddn[t] = 0.f;
        }
        if (k >= 1) {
            const float hoFb = vd_h<float>(ho[(k - 1) * P]), hnFb = vd_h<float>(hn[(k - 1) * P]);
            const float nb = nuh[k * P];
#pragma unroll
            for (int t = 0; t < NT; t++) {
                const float x = dt2 * (nb + mol[t]);
                aob[t] = co * x / (hoF + hoFb);
                anb[t] = cn * x / (hnF + hnFb);
                ddn[t] = inc_f<S>(v[t][(k - 1) * P] - xc[t]);
            }
        }
        // operands of the level above (k + 1), one level ahead of the arithmetic
        double ho_a = 0.0, hn_a = 0.0;
        float nuh_a = 0.f, e2c[NT], e4c[NT];
        S xa[NT];
        if (k + 1 < nz) {
            ho_a = ho[(k + 1) * P];
            hn_a = hn[(k + 1) * P];
            nuh_a = nuh[(k + 1) * P];
        }
#pragma unroll
        for (int t = 0; t < NT; t++) {
            xa[t] = k + 1 < nz ? v[t][(k + 1) * P] : S(0);
            e2c[t] = SRC && e2[t] ? e2[t][k * P] : 0.f;
            e4c[t] = SRC && e4[t] ? e4[t][k * P] : 0.f;
        }
        float L0[NT], D0[NT], U0[NT], R0[NT], al[NT], ga[NT], de[NT];
        for (int ii = 0; ii < m; ii++, k++) {
            const bool top = k == nz - 1, bot = k == 0;
            // raw operands of level k + 2 and the sources of level k + 1
            double ho_n = 0.0, hn_n = 0.0;
            float nuh_n = 0.f, e2n[NT], e4n[NT];
            S xn[NT];
            if (k + 2 < nz) {
                ho_n = ho[(k + 2) * P];
                hn_n = hn[(k + 2) * P];
                nuh_n = nuh[(k + 2) * P];
            }
#pragma unroll
            for (int t = 0; t < NT; t++) {
                xn[t] = k + 2 < nz ? v[t][(k + 2) * P] : S(0);
                e2n[t] = SRC && e2[t] && k + 1 < nz ? e2[t][(k + 1) * P] : 0.f;
                e4n[t] = SRC && e4[t] && k + 1 < nz ? e4[t][(k + 1) * P] : 0.f;
            }
            const float hoFa = top ? 0.f : vd_h<float>(ho_a), hnFa = top ? 0.f : vd_h<float>(hn_a);
            const float dha = (one_h || top) ? 0.f : getm_d2f_approx(ho_a - hn_a);
#pragma unroll
            for (int t = 0; t < NT; t++) {
                // interface above level k (vd_aux with C level k) and the
                // difference to the level above, as in vd_inc_sweep
                float aoa = 0.f, ana = 0.f, dup = 0.f;
                if (!top) {
                    const float x = dt2 * (nuh_a + mol[t]);
                    aoa = co * x / (hoFa + hoF);
                    ana = cn * x / (hnFa + hnF);
                    dup = inc_f<S>(xa[t] - xc[t]);
                }
                const float xk = inc_f<S>(xc[t]);
                float dg, rh;
                if (top) {
                    dg = hnF + anb[t];
                    rh = xk * dh + ddn[t] * (aob[t] + anb[t]);
                } else if (bot) {
                    dg = hnF + ana;
                    rh = xk * dh + dup * (aoa + ana);
                } else {
                    dg = hnF + ana + anb[t];
                    rh = xk * dh + dup * (aoa + ana) + ddn[t] * (aob[t] + anb[t]);
                }
                if (SRC && e2[t]) rh = rh + e2c[t] * xk;
                if (SRC && e2[t]) dg = dg - e2c[t];
                if (SRC && e4[t]) rh = rh + e4c[t];
                const float lw = bot ? 0.f : -anb[t];
                const float up = top ? 0.f : -ana;
                if (ii == 0) {
                    L0[t] = lw; D0[t] = dg; U0[t] = up; R0[t] = rh;
                } else if (ii == 1) {
                    const float inv = 1.f / dg;
                    al[t] = lw * inv; ga[t] = up * inv; de[t] = rh * inv;
                } else {
                    const float inv = 1.f / (dg - lw * ga[t]);
                    al[t] = -(lw * al[t]) * inv;
                    ga[t] = up * inv;
                    de[t] = (rh - lw * de[t]) * inv;
                }
                if (ii >= 1 && ii < m - 1) {
                    VD_ROW(t, 0, ii) = al[t];
                    VD_ROW(t, 1, ii) = ga[t];
                    VD_ROW(t, 2, ii) = de[t];
                }
                aob[t] = aoa; anb[t] = ana; ddn[t] = -dup;
                xc[t] = xa[t]; xa[t] = xn[t];
                e2c[t] = e2n[t]; e4c[t] = e4n[t];
            }
            hoF = hoFa; hnF = hnFa; dh = dha;
            ho_a = ho_n; hn_a = hn_n; nuh_a = nuh_n;
        }
        // down through the inner levels: dx_ii = d - a dx_first - g dx_last
        float as[NT], gs[NT], ds[NT];
#pragma unroll
        for (int t = 0; t < NT; t++) { as[t] = 0.f; gs[t] = -1.f; ds[t] = 0.f; }
        for (int ii = m - 2; ii >= 1; ii--) {
#pragma unroll
            for (int t = 0; t < NT; t++) {
                const float a_ = VD_ROW(t, 0, ii), g_ = VD_ROW(t, 1, ii), d_ = VD_ROW(t, 2, ii);
                ds[t] = d_ - g_ * ds[t];
                as[t] = a_ - g_ * as[t];
                gs[t] = -(g_ * gs[t]);
                VD_ROW(t, 0, ii) = as[t];
                VD_ROW(t, 1, ii) = gs[t];
                VD_ROW(t, 2, ii) = ds[t];
            }
        }
        // the segment's rows of the reduced system
#pragma unroll
        for (int t = 0; t < NT; t++) {
            VD_RED(t, 0, 2 * s) = L0[t];
            VD_RED(t, 1, 2 * s) = D0[t] - U0[t] * as[t];
            VD_RED(t, 2, 2 * s) = -(U0[t] * gs[t]);
            VD_RED(t, 3, 2 * s) = R0[t] - U0[t] * ds[t];
            VD_RED(t, 0, 2 * s + 1) = al[t];
            VD_RED(t, 1, 2 * s + 1) = 1.f;
            VD_RED(t, 2, 2 * s + 1) = ga[t];
            VD_RED(t, 3, 2 * s + 1) = de[t];
        }
    }
    __syncthreads();
    if (s == 0 && act) {
#pragma unroll
        for (int t = 0; t < NT; t++) {
            float cp[R], dp[R];
            cp[0] = VD_RED(t, 2, 0) / VD_RED(t, 1, 0);
            dp[0] = VD_RED(t, 3, 0) / VD_RED(t, 1, 0);
#pragma unroll
            for (int r = 1; r < R; r++) {
                const float lw = VD_RED(t, 0, r);
                const float inv = 1.f / (VD_RED(t, 1, r) - lw * cp[r - 1]);
                cp[r] = VD_RED(t, 2, r) * inv;
                dp[r] = (VD_RED(t, 3, r) - lw * dp[r - 1]) * inv;
            }
            float x = dp[R - 1];
            VD_RED(t, 3, R - 1) = x;
#pragma unroll
            for (int r = R - 2; r >= 0; r--) {
                x = dp[r] - cp[r] * x;
                VD_RED(t, 3, r) = x;
            }
        }
    }
    __syncthreads();
    if (act) {
#pragma unroll
        for (int t = 0; t < NT; t++) {
            S* __restrict__ vt = a.var[t0 + t] + c;
            const float xF = VD_RED(t, 3, 2 * s), xL = VD_RED(t, 3, 2 * s + 1);
            S xo = vt[klo * P];
            for (int ii = 0; ii < m; ii++) {
                const int k = klo + ii;
                const S xnext = ii + 1 < m ? vt[(k + 1) * P] : S(0);
                const float dx = ii == 0 ? xF
                                 : ii == m - 1 ? xL
                                               : VD_ROW(t, 2, ii) - VD_ROW(t, 0, ii) * xF - VD_ROW(t, 1, ii) * xL;
                vt[k * P] = inc_add<S>(xo, dx);
                xo = xnext;
            }
        }
    }
    __syncthreads();  // shared memory is reused by the next group of fields
#undef VD_ROW
#undef VD_RED
}

// One row j of 32 columns per block (blockIdx.x: 32-column strip, blockIdx.y:
// row); fields in groups of NT (then an odd last one alone).
template <int NT, bool SRC, typename S>
__global__ void __launch_bounds__(VD_SEG_THREADS, 4) vd_seg_kernel(VDArgs<float, S> a)
{
    extern __shared__ __align__(16) unsigned char vd_smem[];
    const int tx = threadIdx.x, s = threadIdx.y, tid = s * 32 + tx;
    const int i = blockIdx.x * 32 + tx, j = blockIdx.y;
    const long long c = (long long)j * a.nx_ + i;
    const bool act = i < a.nx_ && a.mask[c] == 1;
    const int nz = a.nz;
    const int klo = s * nz / VD_NSEG, m = (s + 1) * nz / VD_NSEG - klo;
    const int maxm = (nz + VD_NSEG - 1) / VD_NSEG;
    const int slots = maxm > 2 ? maxm - 2 : 0;
    float* rows = (float*)vd_smem;
    float* red = rows + (size_t)3 * NT * slots * VD_SEG_THREADS;
    int t0 = 0;
    for (; t0 + NT <= a.ntracer; t0 += NT) vd_seg_group<NT, SRC, S>(a, c, act, t0, s, klo, m, slots, rows, red, tid, tx);
    if constexpr (NT > 1)
        for (; t0 < a.ntracer; t0++) vd_seg_group<1, SRC, S>(a, c, act, t0, s, klo, m, slots, rows, red, tid, tx);
}

template <int NT, bool SRC, typename S>
static int vd_seg_launch_one(VDArgs<float, S>& a, cudaStream_t stream)
{
    const size_t smem = vd_seg_smem(a.nz, NT);
    if (smem > 48 * 1024) {
        // nz up to VD_NSEG * VD_SEG_MAXM needs at most ~60 KB
        if (cudaFuncSetAttribute(vd_seg_kernel<NT, SRC, S>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)smem) != cudaSuccess)
            return GETM_ERR_CUDA;
    }
    const dim3 grid(getm_div_up(a.nx_, 32), a.ny_), block(32, VD_NSEG);
    vd_seg_kernel<NT, SRC, S><<<grid, block, smem, stream>>>(a);
    GETM_CHECK_LAUNCH();
    return GETM_OK;
}

// Whether the segmented solve takes this call (knob set, nz in range).
static bool vd_seg_applies(int nz)
{
    return getm_tune(GETM_TUNE_COLUMN_SOLVE) == 1 && nz >= 2 * VD_NSEG && nz <= VD_NSEG * VD_SEG_MAXM;
}

template <typename S>
static int vd_seg_launch(VDArgs<float, S>& a, cudaStream_t stream)
{
    bool src = false;
    for (int t = 0; t < a.ntracer; t++) src = src || a.ea2[t] || a.ea4[t];
    const bool pairs = a.ntracer > 1;
    if (src && pairs) return vd_seg_launch_one<2, true, S>(a, stream);
    if (src) return vd_seg_launch_one<1, true, S>(a, stream);
    if (pairs) return vd_seg_launch_one<2, false, S>(a, stream);
    return vd_seg_launch_one<1, false, S>(a, stream);
}

// The increment-form solve for FP64-stored fields (float solve, nuh and
// sources; work: 2 nz planes of floats per field of a pair).
static int vd_launch_f64s(VDArgs<float, double>& a, cudaStream_t stream)
{
    if (a.nz > 1 && vd_seg_applies(a.nz)) return vd_seg_launch(a, stream);
    if (!a.work) return GETM_ERR_ARG;
    return vd_inc_launch(a, stream);
}

// prepare as a separate call (diffusion.F90:163-171): auxo/auxn at every
// point of the halo-inclusive extent, Fortran levels kmin..kmax-1.
__global__ void vd_prepare_kernel(int nx_, int ny_, int nz, long long plane, double molecular,
                                  const double* nuh, double dt, double cnpar, const double* dzo,
                                  const double* dzn, double* auxo, double* auxn)
{
    long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    long long n = plane * (nz - 1);
    if (p >= n) return;
    int k = (int)(p / plane);
    long long c = p - (long long)k * plane;
    double x = 2.0 * dt * (nuh[c + (k + 1) * plane] + molecular);
    auxo[p] = (1.0 - cnpar) * x / (dzo[c + (k + 1) * plane] + dzo[c + k * plane]);
    auxn[p] = cnpar * x / (dzn[c + (k + 1) * plane] + dzn[c + k * plane]);
}

static int vd_launch(VDArgs<float>& a, cudaStream_t stream)
{
    if (a.work && a.nz > 1) {
        if (vd_seg_applies(a.nz)) return vd_seg_launch(a, stream);
        return vd_inc_launch(a, stream);
    }
    int threads = 128;
    const size_t per = (size_t)VD_SMEM_ARRAYS * a.nz * sizeof(float);
    while (threads > 32 && per * threads > 160 * 1024) threads /= 2;
    size_t smem = per * threads;
    if (smem > 200 * 1024) return GETM_ERR_NZ;
    static std::atomic<unsigned long long> done{0};
    if (!getm_once_per_device(done, [] {
            return cudaFuncSetAttribute(vd_column_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024) ==
                   cudaSuccess;
        }))
        return GETM_ERR_CUDA;
    dim3 grid(getm_div_up(a.nx_, threads), a.ny_);
    vd_column_kernel<<<grid, threads, smem, stream>>>(a);
    GETM_CHECK_LAUNCH();
    return GETM_OK;
}

template <bool SRC>
static int vd_f64_launch_one(VDArgs<double>& a, int rows, int nz, size_t smem, cudaStream_t stream)
{
    static std::atomic<unsigned long long> done{0};
    if (smem > 0 && !getm_once_per_device(done, [] {
            return cudaFuncSetAttribute(vd_f64_kernel<SRC>, cudaFuncAttributePreferredSharedMemoryCarveout, 100) ==
                       cudaSuccess &&
                   cudaFuncSetAttribute(vd_f64_kernel<SRC>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        200 * 1024) == cudaSuccess;
        }))
        return GETM_ERR_CUDA;
    const dim3 grid(getm_div_up(a.nx_, 32), getm_div_up(a.ny_, rows), nz), block(32, rows);
    vd_f64_kernel<SRC><<<grid, block, smem, stream>>>(a);
    GETM_CHECK_LAUNCH();
    return GETM_OK;
}

// FP64 form: blocks of fewer rows where four would leave SMs without work (an
// SM's FP64 pipe is the bound, so the columns are spread over all).
static int vd_launch(VDArgs<double> a, cudaStream_t stream)
{
    bool src = false;
    for (int t = 0; t < a.ntracer; t++) src = src || a.ea2[t] || a.ea4[t];
    // The fields of a batch side by side, their coefficients in shared memory
    // instead of the workspace: where that keeps more warps on an SM than one
    // field's columns alone (five blocks' worth, 20, at most), and where the
    // columns do not fit at once (the last wave, of few warps, would take all
    // fields again); up to the layers that leave room for ten warps.  us, fields in
    // turn through the workspace -> side by side: 200 x 150 x 30 two 125 -> 119,
    // 120 x 100 x 30 two 76 -> 53, 92 x 92 x 20 six 162 -> 68, 400 x 300 x 40 two 756
    // -> 558, one 394 -> 319, 400 x 300 x 20 two 365 -> 267; but 300 x 200 x 30
    // three (13 warps of columns, 14 in shared memory) 313 -> 343, 300 x 250 x 64
    // one 342 -> 392.
    const long long strips = getm_div_up(a.nx_, 32);
    const double columns = (double)strips * a.ny_ / GETM_SMS;  // warps per SM
    const double shared = fmin(224.0 * 1024 / (2.0 * a.nz * 32 * sizeof(double)), columns * a.ntracer);
    const bool side = a.nz > 1 && a.nz <= 44 && a.ntracer > 0 && (columns > 20.0 || shared >= 1.25 * columns) &&
                      (a.ntracer == 1 || vd_fields_apart(a));
    const int nz = side ? a.ntracer : 1;
    if (side) a.work = nullptr;
    int rows = 4;
    while (rows > 1 && strips * getm_div_up(a.ny_, rows) * nz < 4 * GETM_SMS) rows /= 2;
    size_t smem = 0;
    if (!a.work && a.nz > 1) {
        const size_t per = (size_t)2 * a.nz * 32 * sizeof(double);  // per row of 32 columns
        while (rows > 1 && per * rows > 160 * 1024) rows /= 2;
        smem = per * rows;
        if (smem > 200 * 1024) return GETM_ERR_NZ;
    }
    return src ? vd_f64_launch_one<true>(a, rows, nz, smem, stream) : vd_f64_launch_one<false>(a, rows, nz, smem, stream);
}

extern "C" int getm_vertical_diffusion_create(getm_grid* tgrid, getm_vertical_diffusion** out)
{
    if (!out) return GETM_ERR_ARG;
    getm_vertical_diffusion* d = (getm_vertical_diffusion*)calloc(1, sizeof(*d));
    if (!d) return GETM_ERR_ALLOC;
    d->tgrid = tgrid;
    *out = d;
    return GETM_OK;
}

extern "C" int getm_vertical_diffusion_finalize(getm_vertical_diffusion* d)
{
    if (!d) return GETM_OK;
    cudaFree(d->auxo);
    cudaFree(d->auxn);
    free(d);
    return GETM_OK;
}

extern "C" int getm_vertical_diffusion_prepare(getm_vertical_diffusion* d, int nx, int ny, int nz,
                                               double molecular, const double* nuh,
                                               double timestep, double cnpar, const int* mask,
                                               const double* ho, const double* hn,
                                               cudaStream_t stream)
{
    (void)mask;
    if (!d || nx < 1 || ny < 1 || nz < 1 || !nuh || !ho || !hn) return GETM_ERR_ARG;
    if (nz > GETM_MAX_NZ) return GETM_ERR_NZ;
    if (nz == 1) return GETM_OK;  // diffusion.F90:155
    const long long plane = (long long)nx * ny;
    const size_t n3 = (size_t)plane * nz;
    if (n3 > d->n3) {
        if (d->auxo) cudaFree(d->auxo);  // (cudaFree waits for the whole device)
        if (d->auxn) cudaFree(d->auxn);
        d->auxo = d->auxn = NULL;
        if (cudaMalloc(&d->auxo, n3 * sizeof(double)) != cudaSuccess) return GETM_ERR_ALLOC;
        if (cudaMalloc(&d->auxn, n3 * sizeof(double)) != cudaSuccess) return GETM_ERR_ALLOC;
        d->n3 = n3;
    }
    long long n = plane * (nz - 1);
    vd_prepare_kernel<<<getm_div_up(n, 256), 256, 0, stream>>>(nx, ny, nz, plane, molecular, nuh, timestep, cnpar, ho, hn, d->auxo, d->auxn);
    GETM_CHECK_LAUNCH();
    return GETM_OK;
}

extern "C" int getm_vertical_diffusion_apply(getm_vertical_diffusion* d, int nx, int ny, int nz,
                                             const int* mask, const double* ho, const double* hn,
                                             double* var, const double* ea2, const double* ea4,
                                             cudaStream_t stream)
{
    if (!d || nx < 1 || ny < 1 || nz < 1 || !mask || !ho || !hn || !var) return GETM_ERR_ARG;
    if (nz > GETM_MAX_NZ) return GETM_ERR_NZ;
    if (nz > 1 && (!d->auxo || d->n3 < (size_t)nx * ny * nz)) return GETM_ERR_ARG;  // not prepared
    VDArgs<double> a;
    memset(&a, 0, sizeof(a));
    a.nx_ = nx; a.ny_ = ny; a.nz = nz; a.plane = (long long)nx * ny;
    a.mask = mask; a.ho = ho; a.hn = hn; a.auxo = d->auxo; a.auxn = d->auxn;
    a.ntracer = 1; a.var[0] = var; a.ea2[0] = ea2; a.ea4[0] = ea4;
    return vd_launch(a, stream);
}

template <typename T, typename S = T>
static int vd_batch_impl(int nx, int ny, int nz, const int* mask, const T* nuh, double timestep, double cnpar,
                         const double* ho, const double* hn, int ntracer, const double* molecular,
                         S* const* vars, const T* const* ea2, const T* const* ea4, T* work, cudaStream_t stream)
{
    if (nx < 1 || ny < 1 || nz < 1 || !mask || !nuh || !ho || !hn || ntracer < 1 || !vars || !molecular)
        return GETM_ERR_ARG;
    if (nz > GETM_MAX_NZ) return GETM_ERR_NZ;
    VDArgs<T, S> a;
    memset(&a, 0, sizeof(a));
    a.nx_ = nx; a.ny_ = ny; a.nz = nz; a.plane = (long long)nx * ny;
    a.mask = mask; a.nuh = nuh; a.ho = ho; a.hn = hn; a.dt = timestep; a.cnpar = cnpar;
    a.work = work;
    int done = 0;
    do {
        int n = ntracer - done;
        if (n > VD_MAX_BATCH) n = VD_MAX_BATCH;
        a.ntracer = n;
        for (int t = 0; t < n; t++) {
            a.molecular[t] = molecular[done + t];
            a.var[t] = vars[done + t];
            a.ea2[t] = ea2 ? ea2[done + t] : NULL;
            a.ea4[t] = ea4 ? ea4[done + t] : NULL;
        }
        int rc;
        if constexpr (std::is_same<T, S>::value) rc = vd_launch(a, stream);
        else rc = vd_launch_f64s(a, stream);
        if (rc) return rc;
        done += n;
    } while (done < ntracer);
    return GETM_OK;
}

extern "C" int getm_vertical_diffusion_batch(int nx, int ny, int nz, const int* mask,
                                             const double* nuh, double timestep, double cnpar,
                                             const double* ho, const double* hn, int ntracer,
                                             const double* molecular, double* const* vars,
                                             const double* const* ea2, const double* const* ea4,
                                             double* work, cudaStream_t stream)
{
    return vd_batch_impl<double>(nx, ny, nz, mask, nuh, timestep, cnpar, ho, hn, ntracer, molecular, vars, ea2, ea4,
                                 work, stream);
}

extern "C" int getm_vertical_diffusion_batch_f32(int nx, int ny, int nz, const int* mask, const float* nuh,
                                                 double timestep, double cnpar, const double* ho,
                                                 const double* hn, int ntracer, const double* molecular,
                                                 float* const* vars, const float* const* ea2,
                                                 const float* const* ea4, float* work, cudaStream_t stream)
{
    return vd_batch_impl<float>(nx, ny, nz, mask, nuh, timestep, cnpar, ho, hn, ntracer, molecular, vars, ea2, ea4,
                                work, stream);
}

extern "C" int getm_vertical_diffusion_batch_f64s(int nx, int ny, int nz, const int* mask, const float* nuh,
                                                  double timestep, double cnpar, const double* ho,
                                                  const double* hn, int ntracer, const double* molecular,
                                                  double* const* vars, const float* const* ea2,
                                                  const float* const* ea4, float* work, cudaStream_t stream)
{
    return vd_batch_impl<float, double>(nx, ny, nz, mask, nuh, timestep, cnpar, ho, hn, ntracer, molecular, vars,
                                        ea2, ea4, work, stream);
}
