// Two-equation (k-epsilon) turbulence closure for sm_103a: the turbulent
// viscosity num and diffusivity nuh at the layer interfaces.
//
// pygetm takes num and nuh from GOTM through pygotm
// (python/pygetm/vertical_mixing.py:60-188, advanced once per 3D step at
// python/pygetm/simulation.py:1107-1115 with ustar_s, ustar_b, z0s, z0b, NN and
// SS).  GOTM is an external package that the reference does not vendor, so
// this is not its code: it is the buoyancy-extended k-epsilon model of Rodi
// (1987, J. Geophys. Res. 92, "Examples of calculation methods for flow and
// mixing in stratified fluids") with constant stability functions, the
// standard model constants (Launder and Spalding 1974), log-law (Dirichlet)
// boundary values for k and epsilon at the bottom and surface interfaces,
// the length-scale limitation of Galperin et al. (1988) in stable
// stratification, and the source-term linearisation of Patankar (1980)
// that keeps k and epsilon positive in the implicit update:
//
//   dk/dt   = d/dz (num/sk dk/dz) + P + B - eps
//   deps/dt = d/dz (num/se deps/dz) + eps/k (c1 P + c3 B - c2 eps)
//   P = num SS, B = -nuh NN, num = cmu k^2/eps, nuh = num / Prt
//
// One thread per water column (32 columns of a warp are adjacent at every
// level, so each level's loads are coalesced); both equations are solved
// implicitly in time over the interfaces 1..nz-1 with an elimination whose
// coefficients live in a [level][column] workspace.  GB300's FP64 rate bounds
// it, so it counts FP64 instructions: with U = dt K / h the coupling through a
// layer, which is the one above an interface and then the one below the next,
// and s' = 1 - c' of the interface below (the fixed bottom value: c' = 0, s' = 1),
//     t = dz (1 - dt S) + U' s',  den = t + U,  c = U / den,  s = t / den,
//     d = (dz (x + dt Q) + U' d') / den,   then downwards x = d + c x_above:
// no large terms are subtracted (b - a c of the textbook form loses digits
// where mixing is strong), one reciprocal per interface (getm_rcp) and one per
// layer, and minima, maxima and comparisons on the integer pipe: about 85 per
// level for both equations and the closure, where 18 divisions and square
// roots alone took some 160.  The operands of a level are loaded a level
// ahead.  200 x 150 x 30: 464 -> 215 us.
#include "getm_common.cuh"

namespace {

// R: type of NN, SS, num and nuh (float in the mixed form); k, epsilon and
// L are FP64 in both forms, and so is the arithmetic.
template <typename R>
struct KepsArgs {
    int nx, ny, nz;
    long long plane;
    int ilo, ihi, jlo, jhi;
    const int* mask;
    const double* h;  // layer thicknesses, nz layers
    const double *ustar_s, *ustar_b, *z0s, *z0b;
    const R *NN, *SS;  // nz + 1 interfaces
    double *tke, *eps, *L;
    R *num, *nuh;
    double* work;  // 2 (nz + 1) planes
    double dt;
    getm_keps_params p;
};

// log-law boundary values at the interface at distance z0 from the wall
__device__ __forceinline__ void keps_wall(const getm_keps_params& p, double ustar, double z0, double& k, double& e)
{
    const double cm0 = p.cm0;
    k = fmax(ustar * ustar / (cm0 * cm0), p.k_min);
    e = fmax(cm0 * cm0 * cm0 * k * sqrt(k) / (p.kappa * z0), p.eps_min);
}

// The operands of interface l (1..nz-1) and of the layer above it.
struct KepsIn {
    double h, num, nuh, SS, NN, k, e;
};

template <typename R>
__device__ __forceinline__ KepsIn keps_load(const KepsArgs<R>& a, long long q)
{
    return KepsIn{a.h[q], getm_widen(a.num[q]), getm_widen(a.nuh[q]), getm_widen(a.SS[q]), getm_widen(a.NN[q]),
                  a.tke[q], a.eps[q]};
}

// One implicit diffusion-source equation over interfaces 1..nz-1 of column c:
// dz_i (x_i' - x_i) / dt = flux differences + dz_i (Q_i + S_i x_i'), S <= 0,
// diffusivities at the layers (between interfaces) the mean of num over sigma,
// Dirichlet values x0, xn at interfaces 0 and nz.  src(in, x, Q, S): the old
// value and the sources; fin(x): the new value's bound.  (x is a.tke or a.eps,
// which keps_load reads: not restrict)
template <typename R, typename Src, typename Fin>
__device__ __forceinline__ void keps_solve(const KepsArgs<R>& a, long long c, double* x, double sigma,
                                           double x0, double xn, Src src, Fin fin)
{
    const long long P = a.plane;
    const int nz = a.nz;
    double* __restrict__ cp = a.work + c;
    double* __restrict__ dp = a.work + (long long)(nz + 1) * P + c;
    const double dts = 0.5 * a.dt / sigma;  // coupling of a layer: dts (num below + num above) / h
    const double numb = getm_widen(a.num[c]);
    double hb = a.h[c];  // layer below interface i
    KepsIn in = keps_load(a, c + P);
    double U = dts * (numb + in.num) * getm_rcp(hb);
    double s = 1.0, d = x0;  // (interface 0 is fixed: c = 0)
    for (int i = 1; i < nz; i++) {
        const long long q = c + (long long)i * P;
        // interface i + 1 (its num and, but for the last, the rest)
        KepsIn nx;
        if (i + 1 < nz) nx = keps_load(a, q + P);
        else nx.num = getm_widen(a.num[q + P]);
        const double dz = getm_half(hb + in.h);
        double xo, Q, S;
        src(in, xo, Q, S);
        const double Un = dts * (in.num + nx.num) * getm_rcp(in.h);
        const double t = fma(U, s, dz * fma(-a.dt, S, 1.0));
        const double r = getm_rcp(t + Un);
        const double cc = Un * r;
        // an infinite sink (S of a zero kinetic energy) fixes the value at zero, as
        // a boundary would: c = 0, s = 1
        s = ((__double2hiint(r) & 0x7fffffff) | __double2loint(r)) != 0 ? t * r : 1.0;
        double rhs = fma(U, d, dz * fma(a.dt, Q, xo));
        // the surface value's coupling enters here and once more in the substitution,
        // which starts from xn with c as it is: it counts twice, as in the oracle
        if (i == nz - 1) rhs = fma(Un, xn, rhs);
        d = rhs * r;
        cp[(long long)i * P] = cc;
        dp[(long long)i * P] = d;
        hb = in.h;
        U = Un;
        in = nx;
    }
    double xv = xn;
    double cn = cp[(long long)(nz - 1) * P], dn = dp[(long long)(nz - 1) * P];
    for (int i = nz - 1; i >= 1; i--) {
        const double cc = cn, dd = dn;
        if (i > 1) {
            cn = cp[(long long)(i - 1) * P];
            dn = dp[(long long)(i - 1) * P];
        }
        xv = fma(cc, xv, dd);
        x[c + (long long)i * P] = fin(xv);
    }
    x[c] = x0;
    x[c + (long long)nz * P] = xn;
}

template <typename R>
__global__ void __launch_bounds__(128) keps_kernel(KepsArgs<R> a)
{
    const int i = blockIdx.x * 32 + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    if (i < a.ilo || i > a.ihi || j < a.jlo || j > a.jhi) return;
    const long long c = (long long)j * a.nx + i;
    if (a.mask[c] != 1) return;
    const getm_keps_params& p = a.p;
    const long long P = a.plane;
    const int nz = a.nz;
    const double cmu = p.cm0 * p.cm0 * p.cm0 * p.cm0;
    const double cde = p.cm0 * p.cm0 * p.cm0;
    double kb, eb, ks, es;
    keps_wall(p, a.ustar_b[c], a.z0b[c], kb, eb);
    keps_wall(p, a.ustar_s[c], a.z0s[c], ks, es);

    // turbulent kinetic energy (old epsilon and diffusivities in the sources)
    auto src_k = [&](const KepsIn& in, double& x, double& Q, double& S) {
        const double prod = in.num * in.SS, buoy = -in.nuh * in.NN;
        const double sum = prod + buoy;
        const bool up = getm_positive_i(sum);
        x = in.k;
        Q = up ? sum : prod;
        S = -getm_div(up ? in.e : in.e - buoy, in.k);
    };
    // (the forward sweep reads every old value before the back substitution
    // overwrites them, so the update is in place)
    keps_solve(a, c, a.tke, p.sig_k, kb, ks, src_k, [&](double x) { return getm_fmax_i(x, p.k_min); });

    // dissipation rate (sources from the new k and the old epsilon)
    auto src_e = [&](const KepsIn& in, double& x, double& Q, double& S) {
        const double prod = in.num * in.SS, buoy = -in.nuh * in.NN;
        const double r = getm_div(in.e, in.k);
        const double c3 = getm_positive_i(buoy) ? p.c3_plus : p.c3_minus;
        x = in.e;
        Q = r * fma(p.c1, prod, c3 * buoy);
        S = -p.c2 * r;
    };
    keps_solve(a, c, a.eps, p.sig_e, eb, es, src_e, [](double x) { return x; });

    // limits, length scale, viscosity and diffusivity at every interface
    const double ilim = cde / p.galp, iprandtl = 1.0 / p.prandtl;
    const bool one = p.prandtl == 1.0;
    double kn = a.tke[c], en = a.eps[c], N2n = getm_widen(a.NN[c]);
    for (int l = 0; l <= nz; l++) {
        const long long q = c + (long long)l * P;
        const double k = kn, N2 = N2n;
        double e = getm_fmax_i(en, p.eps_min);
        if (l < nz) {
            kn = a.tke[q + P];
            en = a.eps[q + P];
            N2n = getm_widen(a.NN[q + P]);
        }
        // Galperin: L = cde k^1.5 / eps <= galp sqrt(2 k / N2)
        if (l > 0 && l < nz && getm_positive_i(N2)) e = getm_fmax_i(e, ilim * k * sqrt(getm_half(N2)));
        a.eps[q] = e;
        const double kr = k * getm_rcp(e);
        a.L[q] = cde * kr * sqrt(k);
        const double nu = cmu * k * kr;
        a.num[q] = (R)nu;
        a.nuh[q] = (R)(one ? nu : nu * iprandtl);
    }
}

}  // namespace

extern "C" int getm_keps_default_params(getm_keps_params* p)
{
    if (!p) return GETM_ERR_ARG;
    p->cm0 = 0.5477;
    p->kappa = 0.4;
    p->sig_k = 1.0;
    p->sig_e = 1.3;
    p->c1 = 1.44;
    p->c2 = 1.92;
    p->c3_minus = -0.4;
    p->c3_plus = 1.0;
    p->galp = 0.53;
    p->prandtl = 1.0;
    p->k_min = 1e-10;
    p->eps_min = 1e-12;
    return GETM_OK;
}

template <typename R>
static int keps_impl(int nx, int ny, int nz, int halox, int haloy, const getm_keps_params* params, double timestep,
                     const int* mask, const double* h, const double* ustar_s, const double* ustar_b,
                     const double* z0s, const double* z0b, const R* NN, const R* SS, double* tke, double* eps,
                     double* L, R* num, R* nuh, double* work, cudaStream_t stream)
{
    if (nx < 1 || ny < 1 || nz < 2 || halox < 0 || haloy < 0 || !params || !(timestep > 0.0)) return GETM_ERR_ARG;
    const void* ptrs[] = {mask, h, ustar_s, ustar_b, z0s, z0b, NN, SS, tke, eps, L, num, nuh, work};
    for (const void* q : ptrs)
        if (!q) return GETM_ERR_ARG;
    KepsArgs<R> a;
    a.nx = nx; a.ny = ny; a.nz = nz; a.plane = (long long)nx * ny;
    a.ilo = halox; a.ihi = nx - halox - 1; a.jlo = haloy; a.jhi = ny - haloy - 1;
    a.mask = mask; a.h = h; a.ustar_s = ustar_s; a.ustar_b = ustar_b; a.z0s = z0s; a.z0b = z0b;
    a.NN = NN; a.SS = SS; a.tke = tke; a.eps = eps; a.L = L; a.num = num; a.nuh = nuh; a.work = work;
    a.dt = timestep;
    a.p = *params;
    const dim3 grid(getm_div_up(nx, 32), getm_div_up(ny, 4)), block(32, 4);
    keps_kernel<R><<<grid, block, 0, stream>>>(a);
    GETM_CHECK_LAUNCH();
    return GETM_OK;
}

extern "C" int getm_keps_advance(int nx, int ny, int nz, int halox, int haloy, const getm_keps_params* params,
                                 double timestep, const int* mask, const double* h, const double* ustar_s,
                                 const double* ustar_b, const double* z0s, const double* z0b, const double* NN,
                                 const double* SS, double* tke, double* eps, double* L, double* num, double* nuh,
                                 double* work, cudaStream_t stream)
{
    return keps_impl<double>(nx, ny, nz, halox, haloy, params, timestep, mask, h, ustar_s, ustar_b, z0s, z0b, NN, SS,
                             tke, eps, L, num, nuh, work, stream);
}

extern "C" int getm_keps_advance_f32(int nx, int ny, int nz, int halox, int haloy, const getm_keps_params* params,
                                     double timestep, const int* mask, const double* h, const double* ustar_s,
                                     const double* ustar_b, const double* z0s, const double* z0b, const float* NN,
                                     const float* SS, double* tke, double* eps, double* L, float* num, float* nuh,
                                     double* work, cudaStream_t stream)
{
    return keps_impl<float>(nx, ny, nz, halox, haloy, params, timestep, mask, h, ustar_s, ustar_b, z0s, z0b, NN, SS,
                            tke, eps, L, num, nuh, work, stream);
}
