// Shared device/host helpers for the getm_gb300 CUDA library (sm_103a).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

#include <type_traits>

#include "getm_gb300.h"

// Physical constants of python/src/wrapper.F90:11-13 (module pygetm).
#define GETM_RHO0 1025.0
#define GETM_KAPPA 0.4
#define GETM_G 9.81

// SMs of a GB300: the unit in which grids are made large enough
#define GETM_SMS 152

// Grid handle: index extent plus device pointers to the static metrics that
// the reference reads from its type_getm_grid (src/domain/domain.F90:85-140)
// inside advection_uv_calculate / c_momentum_diffusion.
struct getm_grid {
    int imin, imax, jmin, jmax, kmin, kmax;  // Fortran 1-based interior bounds
    int halox, haloy;
    int nx_, ny_;                            // full extents incl. halos
    const int* mask;
    const double* dx;
    const double* dy;
    const double* idx;
    const double* idy;
    const double* iarea;
    const double* area;
    // float copies of the metrics for the mixed form, built on first use by
    // getm_grid_f32_metrics (device memory owned by the handle)
    float* dx_f;
    float* dy_f;
    float* idx_f;
    float* idy_f;
    float* iarea_f;
};

// Build the float metric copies of a grid if they do not exist yet (one
// cudaMalloc per array and a conversion kernel on `stream`, synchronised with
// the whole device before and after); returns a GETM_* status.  The first
// mixed-form call on a grid makes them, so that call must precede any stream
// capture.
int getm_grid_f32_metrics(getm_grid* g, cudaStream_t stream);

// Launch-shape knob of the calling host thread (GETM_TUNE_*; getm_tune_set).
int getm_tune(int knob);

// Host-side count of kernel launches issued by this library (one increment
// per launch site executed); read with getm_launch_count().
extern "C" unsigned long long getm_launch_counter_add(void);

#define GETM_CHECK_LAUNCH()                                     \
    do {                                                        \
        getm_launch_counter_add();                              \
        cudaError_t e_ = cudaGetLastError();                    \
        if (e_ != cudaSuccess) return GETM_ERR_CUDA;            \
    } while (0)

// Sets a kernel's attributes once per device (they belong to the device that is
// current): done holds a bit per device, set(), which may run twice in two
// threads, returns whether it succeeded.
template <typename F>
static inline bool getm_once_per_device(std::atomic<unsigned long long>& done, F set)
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return false;
    const unsigned long long bit = dev < 64 ? 1ull << dev : 0ull;
    if (done.load() & bit) return true;
    if (!set()) return false;
    done.fetch_or(bit);
    return true;
}

static inline unsigned int getm_div_up(long long a, long long b) { return (unsigned int)((a + b - 1) / b); }

// Thread-per-column kernels launched over a flattened range of rows: thread
// t of a 1D grid takes column (j0 + t / width, t % width) of rows j0 ..
// j0 + nrows - 1 (consecutive threads, consecutive points, rows back to back,
// so every block is full whatever the row length); false past the last
// column.  Launch getm_div_up(width * nrows, threads) blocks.
__device__ __forceinline__ bool getm_flat_column(int width, int j0, int nrows, int& i, int& j)
{
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)width * nrows) return false;
    const int r = (int)(t / width);
    j = j0 + r;
    i = (int)(t - (long long)r * width);
    return true;
}

// ---------------------------------------------------------------------------
// double <-> float conversions on the integer pipe.  GB300 runs FP64
// instructions, conversions between double and float included, at a small
// fraction of its FP32/integer rate, so the mixed form's kernels convert the
// FP64 thickness fields by rearranging IEEE-754 bit fields instead.
// getm_f2d: exact float -> double for normal numbers and zeros.
// getm_d2f_approx: double -> float with the mantissa truncated to 23 bits
// (relative error below 2^-23; used only where a float approximation of a
// thickness is needed, e.g. as a divisor of an increment), for doubles in the
// normal float range.  Values outside those ranges take the hardware path.
// ---------------------------------------------------------------------------
// Out-of-line fallbacks: keeping the hardware conversions out of the common
// path stops the compiler from issuing them predicated on every call.
static __device__ __noinline__ double getm_f2d_hw(float x) { return (double)x; }
static __device__ __noinline__ float getm_d2f_hw(double x) { return (float)x; }

// Both work on 32-bit words (one funnel shift carries the three mantissa or
// exponent bits across) with one range test: about half the instructions of
// the 64-bit form, with the same bits.  The mixed kernels issue mostly these:
// 400 x 300 x 40, two tracers, five-pass split 702 -> 649 us, column solve 188 -> 133
// us, one substep 71 -> 67 us.
__device__ __forceinline__ double getm_f2d(float x)
{
    const unsigned int b = __float_as_uint(x);
    if ((b << 1) - (1u << 24) < (254u << 24))  // normal: exponent field 1 .. 254
        return __hiloint2double((int)(((b & 0x7fffffffu) >> 3) + (896u << 20) | (b & 0x80000000u)), (int)(b << 29));
    if ((b << 1) == 0u) return __hiloint2double((int)b, 0);  // signed zero
    return getm_f2d_hw(x);                                   // subnormal, inf, nan
}

__device__ __forceinline__ float getm_d2f_approx(double x)
{
    const unsigned int hi = (unsigned int)__double2hiint(x), lo = (unsigned int)__double2loint(x);
    // exponent field 897 .. 1150: a normal float (exponent less 896, whose
    // multiples of 2^32 fall out of the shifted word)
    if ((hi & 0x7fffffffu) - (897u << 20) < (254u << 20))
        return __uint_as_float((__funnelshift_l(lo, hi, 3) + 0x40000000u & 0x7fffffffu) | (hi & 0x80000000u));
    if (((hi << 1) | lo) == 0u) return __uint_as_float(hi);  // signed zero
    return getm_d2f_hw(x);                                   // outside the normal float range
}

// Increment-form helpers for a field stored as S (float, or double for the
// FP64 storage of the mixed form's 2D momentum and tracers): a value or a
// difference of neighbouring values (formed in S) narrowed to the float
// arithmetic of the increments, and a float increment added in S.
template <typename S>
__device__ __forceinline__ float inc_f(S x)
{
    if constexpr (std::is_same<S, double>::value) return getm_d2f_approx(x);
    else return x;
}

template <typename S>
__device__ __forceinline__ S inc_add(S x, float dx)
{
    if constexpr (std::is_same<S, double>::value) return x + getm_f2d(dx);
    else return x + dx;
}

// A value of the storage type T widened to double: float on the integer pipe
// (getm_f2d, exact), double as it is.
template <typename T>
__device__ __forceinline__ double getm_widen(T x)
{
    if constexpr (std::is_same<T, float>::value) return getm_f2d(x);
    else return x;
}

// x * 2^-n (n = 1, 2) on the integer pipe: exact, and bitwise the FP64
// multiply's result, for normal x whose product stays normal (the exponent
// field decreases by n); zeros, subnormals, infinities and NaNs take the FP64
// multiply out of line (so that it is not issued predicated on every call).
static __device__ __noinline__ double getm_scale_hw(double x, double f) { return x * f; }

template <int N>
__device__ __forceinline__ double getm_pow2_scale_down(double x)
{
    static_assert(N == 1 || N == 2, "halving or quartering");
    const int hi = __double2hiint(x);
    if (((unsigned int)hi & 0x7fffffffu) - ((N + 1u) << 20) < ((0x7ffu - (N + 1u)) << 20))  // N < exponent < 0x7ff
        return __hiloint2double(hi - (N << 20), __double2loint(x));
    return getm_scale_hw(x, N == 1 ? 0.5 : 0.25);
}

__device__ __forceinline__ double getm_half(double x) { return getm_pow2_scale_down<1>(x); }
__device__ __forceinline__ double getm_quarter(double x) { return getm_pow2_scale_down<2>(x); }

// The rest x - getm_f2d(getm_d2f_approx(x)) as a float, on the integer pipe:
// the truncated head keeps the top 24 significant bits of x, so the rest is
// the low 29 bits of the mantissa at the scale of x's last bit (rounded to 24
// bits by the conversion).  |x| below 2^-74 or beyond the float range: the
// FP64 subtraction.
__device__ __forceinline__ float getm_d2f_rest(double x)
{
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    const int e = (int)((b >> 52) & 0x7ffu) - 1023;
    if (e < -74 || e > 127) return getm_d2f_approx(x - getm_f2d(getm_d2f_approx(x)));
    const float r = __uint2float_rn((unsigned int)b & 0x1fffffffu) * __uint_as_float((unsigned int)(e + 75) << 23);
    return (b >> 63) ? -r : r;
}

// Comparisons of doubles on the integer pipe, for the mixed form: GB300
// issues an FP64 instruction (compare, min and max included) at a small
// fraction of the integer rate, and these give the same values.
// getm_dkey maps a double to a signed 64-bit key whose order is the numeric
// order of all non-NaN doubles (-0 orders below +0): the magnitude bits of
// a negative value are inverted.
__device__ __forceinline__ long long getm_dkey(double x)
{
    const long long b = __double_as_longlong(x);
    return b ^ (long long)((unsigned long long)(b >> 63) >> 1);
}

__device__ __forceinline__ bool getm_isnan_i(double x)
{
    return ((unsigned long long)__double_as_longlong(x) << 1) > (0x7ff0000000000000ull << 1);
}

// fmax / fmin semantics (a NaN operand yields the other one)
__device__ __forceinline__ double getm_fmax_i(double a, double b)
{
    if (getm_isnan_i(a)) return b;
    if (getm_isnan_i(b)) return a;
    return getm_dkey(a) >= getm_dkey(b) ? a : b;
}

__device__ __forceinline__ double getm_fmin_i(double a, double b)
{
    if (getm_isnan_i(a)) return b;
    if (getm_isnan_i(b)) return a;
    return getm_dkey(a) <= getm_dkey(b) ? a : b;
}

// x > 0.0 (false for NaN)
__device__ __forceinline__ bool getm_positive_i(double x)
{
    const long long b = __double_as_longlong(x);
    return b > 0 && b <= 0x7ff0000000000000ll;
}

// num / den in FP64 to about 2^-46 relative (not correctly rounded), for the
// mixed form: the float reciprocal of den refined by one Newton-Raphson step
// (q0 = num r, q = q0 + r (num - q0 den)), three FP64 instructions instead of
// a correctly rounded division.  den zero, not finite or outside the normal
// float range: the correctly rounded division.
__device__ __forceinline__ double getm_div_refined(double num, double den)
{
    const float df = getm_d2f_approx(den);
    const float adf = fabsf(df);
    if (!(adf > 1e-30f && adf < 1e30f)) return num / den;
    const double r = getm_f2d(__frcp_rn(df));
    const double q0 = num * r;
    return fma(fma(-q0, den, num), r, q0);
}

// 1 / x in FP64 to within two units in the last place with three FP64
// instructions: the approximate reciprocal r of PTX (rcp.approx.ftz.f64,
// relative error e about 2^-20, not on the FP64 pipe) and one third-order
// Householder step (Householder 1970, The Numerical Treatment of a Single
// Nonlinear Equation), r (1 + e + e^2) with e = 1 - x r, whose own error is e^3.
// GB300 runs FP64 at 1/64 of its float rate and the correctly rounded
// division takes several times as many FP64 instructions, so this serves
// where a quotient only scales an increment.  Zero, subnormal, huge and
// non-finite x: the correctly rounded division, out of line.
static __device__ __noinline__ double getm_rcp_hw(double x) { return 1.0 / x; }

__device__ __forceinline__ double getm_rcp(double x)
{
    const unsigned e11 = ((unsigned)__double2hiint(x) >> 20) & 0x7ffu;
    if (e11 - 2u > 2042u) return getm_rcp_hw(x);  // outside 2^-1021 .. 2^1022
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    const double e = __fma_rn(-x, r, 1.0);
    return __fma_rn(r, __fma_rn(e, e, e), r);
}

// n / d in FP64 with six FP64 instructions: n getm_rcp(d) and one correction by
// its own remainder, formed exactly by a fused multiply-add (Markstein 1990, IBM
// J. Res. Dev. 34, 111-119), which leaves an error of half a unit in the last
// place and less than 2^-6 of one beside it (the correctly rounded division
// takes about twice as many).  Operands or quotients near the ends of the range,
// infinities and NaNs: the division, out of line.
static __device__ __noinline__ double getm_div_hw(double n, double d) { return n / d; }

__device__ __forceinline__ double getm_div(double n, double d)
{
    const int en = (int)(((unsigned)__double2hiint(n) >> 20) & 0x7ffu);
    const int ed = (int)(((unsigned)__double2hiint(d) >> 20) & 0x7ffu);
    const bool zero = ((__double2hiint(n) & 0x7fffffff) | __double2loint(n)) == 0;
    // both within 2^-959 .. 2^960, the quotient within 2^-900 .. 2^900
    if ((unsigned)(ed - 64) > 1919u || (!zero && ((unsigned)(en - 64) > 1919u || (unsigned)(en - ed + 900) > 1800u)))
        return getm_div_hw(n, d);
    const double r = getm_rcp(d);
    const double q = __dmul_rn(n, r);
    return zero ? q : __fma_rn(__fma_rn(-q, d, n), r, q);  // (a signed zero keeps its sign)
}

// 2 x on the integer pipe (exact; zeros, subnormals, infinities, NaNs and
// overflow take the FP64 sum out of line)
static __device__ __noinline__ double getm_twice_hw(double x) { return x + x; }

__device__ __forceinline__ double getm_twice(double x)
{
    const int hi = __double2hiint(x);
    if ((((unsigned)hi >> 20) & 0x7ffu) - 1u < 0x7fdu) return __hiloint2double(hi + (1 << 20), __double2loint(x));
    return getm_twice_hw(x);
}

// x, negated where neg is set, on the integer pipe
__device__ __forceinline__ double getm_negate_if(double x, bool neg)
{
    return __hiloint2double(__double2hiint(x) ^ (neg ? (int)0x80000000 : 0), __double2loint(x));
}

// min and max of non-negative doubles (their bit patterns order as integers)
__device__ __forceinline__ double getm_min_pos(double a, double b)
{
    return __double_as_longlong(a) < __double_as_longlong(b) ? a : b;
}

__device__ __forceinline__ double getm_max_pos(double a, double b)
{
    return __double_as_longlong(a) > __double_as_longlong(b) ? a : b;
}

// True for the mixed form's float bulk type.  Its update kernels use the
// increment form x_new = x_old + dx, with dx formed from small differences,
// so a field that does not change is reproduced exactly and float32 rounding
// scales with the change rather than with the field.  (The FP64 form's advection
// and column solves work in increments too, in FP64 throughout.)
template <typename T>
constexpr bool getm_increment_form = std::is_same<T, float>::value;

// ---------------------------------------------------------------------------
// TVD limiter (src/operators/advection_schemes/limiters.h:1-44).  T is the
// arithmetic type: double for the FP64 form, float for the mixed form.
// ---------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ T getm_limiter(int scheme, T ratio, T cfl)
{
    T limiter;
    switch (scheme) {
    case GETM_SCHEME_HSIMT: {
        T kappa = T(1) - cfl;
        T x = T(0.25) * (kappa - T(1.0) / T(3.0) / kappa);
        limiter = (T(0.5) + x) + (T(0.5) - x) * ratio;
        limiter = fmax(T(0), limiter);
        limiter = fmin(fmin(T(2) * ratio, limiter), T(2));
        break;
    }
    case GETM_SCHEME_MUSCL:
        limiter = fmin(fmin(T(2) * ratio, T(0.5) * (T(1) + ratio)), T(2));
        break;
    case GETM_SCHEME_P2_PDM: {
        T x = T(1.0) / T(6.0) * (T(1) - T(2) * cfl);
        limiter = (T(0.5) + x) + (T(0.5) - x) * ratio;
        limiter = fmin(fmin(T(2) * ratio / (cfl + T(1.e-10)), limiter), T(2) / (T(1) - cfl));
        break;
    }
    case GETM_SCHEME_SPLMAX13:
        limiter = fmin(fmin(T(2) * ratio, T(1.0) / T(3.0) * fmax(T(1) + T(2) * ratio, T(2) + ratio)), T(2));
        break;
    case GETM_SCHEME_SUPERBEE:
        limiter = fmax(fmin(T(2) * ratio, T(1)), fmin(ratio, T(2)));
        break;
    default:
        limiter = T(0);
        break;
    }
    return limiter;
}

// The limited deviation without a division per field (C: float for the mixed
// form, double for the FP64 form).  For deltaf and deltafu of the same sign s,
// phi(r) deltaf with r = deltafu / deltaf equals s phi_a(a, b), a = |deltaf|,
// b = |deltafu|, where phi_a is the limiter's expression with r replaced by b
// and every constant term multiplied by a (all five limiters are piecewise
// linear in r).  The terms that depend only on the Courant number are formed
// once per face (getm_tvd_face_c) and shared by every field advected through
// the face.
template <typename C>
struct TvdFace {
    int scheme;
    C half1mc;     // 0.5 (1 - cfl)
    C lin0, lin1;  // HSIMT, P2_PDM: phi = lin0 + lin1 r
    C rcoef, cap;  // P2_PDM: 2 / (cfl + 1e-10), 2 / (1 - cfl)
};

// Both forms: every product and sum rounded as written (intrinsics where the
// compiler could contract), so that all kernels that share these functions, and
// every shape of one kernel, give the same bits.
__device__ __forceinline__ TvdFace<float> getm_tvd_face_c(int scheme, float cfl)
{
    TvdFace<float> f;
    f.scheme = scheme;
    f.half1mc = 0.5f * __fadd_rn(1.f, -cfl);
    f.lin0 = f.lin1 = 0.f;
    f.rcoef = f.cap = 2.f;
    if (scheme == GETM_SCHEME_HSIMT) {
        const float kappa = __fadd_rn(1.f, -cfl);
        const float x = 0.25f * (kappa - 1.f / 3.f / kappa);  // (0.25 is exact)
        f.lin0 = 0.5f + x;
        f.lin1 = 0.5f - x;
    } else if (scheme == GETM_SCHEME_P2_PDM) {
        const float t = __fmaf_rn(-2.f, cfl, 1.f);
        f.lin0 = __fmaf_rn(1.f / 6.f, t, 0.5f);
        f.lin1 = __fmaf_rn(-1.f / 6.f, t, 0.5f);
        f.rcoef = 2.f / __fadd_rn(cfl, 1.e-10f);
        f.cap = 2.f / __fadd_rn(1.f, -cfl);
    }
    return f;
}

__device__ __forceinline__ TvdFace<double> getm_tvd_face_c(int scheme, double cfl)
{
    TvdFace<double> f;
    f.scheme = scheme;
    f.half1mc = __fma_rn(-0.5, cfl, 0.5);
    f.lin0 = f.lin1 = 0.0;
    f.rcoef = f.cap = 2.0;
    if (scheme == GETM_SCHEME_HSIMT) {
        const double kappa = __dadd_rn(1.0, -cfl);
        const double x = __dmul_rn(0.25, __fma_rn(-1.0 / 3.0, getm_rcp(kappa), kappa));
        f.lin0 = __dadd_rn(0.5, x);
        f.lin1 = __dadd_rn(0.5, -x);
    } else if (scheme == GETM_SCHEME_P2_PDM) {
        const double x = __fma_rn(-1.0 / 3.0, cfl, 1.0 / 6.0);
        f.lin0 = __dadd_rn(0.5, x);
        f.lin1 = __dadd_rn(0.5, -x);
        f.rcoef = __dmul_rn(2.0, getm_rcp(__dadd_rn(cfl, 1.e-10)));
        f.cap = __dmul_rn(2.0, getm_rcp(__dadd_rn(1.0, -cfl)));
    }
    return f;
}

__device__ __forceinline__ float getm_tvd_dev_c(const TvdFace<float>& tf, float deltaf, float deltafu)
{
    if (!(deltaf * deltafu > 0.f)) return 0.f;
    const float a = fabsf(deltaf), b = fabsf(deltafu);
    float pa;
    switch (tf.scheme) {
    case GETM_SCHEME_HSIMT:
        pa = fminf(fminf(2.f * b, fmaxf(0.f, __fmaf_rn(tf.lin0, a, __fmul_rn(tf.lin1, b)))), 2.f * a);
        break;
    case GETM_SCHEME_MUSCL: pa = fminf(fminf(2.f * b, 0.5f * (a + b)), 2.f * a); break;
    case GETM_SCHEME_P2_PDM:
        pa = fminf(fminf(tf.rcoef * b, __fmaf_rn(tf.lin0, a, __fmul_rn(tf.lin1, b))), tf.cap * a);
        break;
    case GETM_SCHEME_SPLMAX13: pa = fminf(fminf(2.f * b, 1.f / 3.f * fmaxf(a + 2.f * b, 2.f * a + b)), 2.f * a); break;
    case GETM_SCHEME_SUPERBEE: pa = fmaxf(fminf(2.f * b, a), fminf(b, 2.f * a)); break;
    default: pa = 0.f; break;
    }
    return tf.half1mc * copysignf(pa, deltaf);
}

// FP64: the limited difference phi(r) deltaf itself, without the factor
// half1mc; signs, doublings, minima and maxima on the integer pipe (superbee
// needs no FP64 instruction at all).  Differences of opposite signs give zero,
// and where one of them is zero every limiter does.  Infinities and NaNs go
// through the ratio, out of line, with the Courant number that half1mc holds
// (times the face's transport QU, as hx_tvd leaves it).
static __device__ __noinline__ double getm_tvd_phi_hw(int scheme, double half1mc, double QU, double deltaf, double deltafu)
{
    const double cfl = QU != 0.0 ? 1.0 - 2.0 * half1mc / QU : 0.0;
    return deltaf * deltafu > 0.0 ? getm_limiter<double>(scheme, deltafu / deltaf, cfl) * deltaf : 0.0;
}

__device__ __forceinline__ double getm_tvd_phi(const TvdFace<double>& tf, double QU, double deltaf, double deltafu)
{
    const int hd = __double2hiint(deltaf), hu = __double2hiint(deltafu);
    const int ha = hd & 0x7fffffff, hb = hu & 0x7fffffff;
    if (ha >= 0x7ff00000 || hb >= 0x7ff00000) return getm_tvd_phi_hw(tf.scheme, tf.half1mc, QU, deltaf, deltafu);
    if ((hd ^ hu) < 0) return 0.0;
    const double a = __hiloint2double(ha, __double2loint(deltaf)), b = __hiloint2double(hb, __double2loint(deltafu));
    double pa;
    switch (tf.scheme) {
    case GETM_SCHEME_HSIMT: {
        const double lin = __fma_rn(tf.lin1, b, __dmul_rn(tf.lin0, a));
        pa = getm_min_pos(getm_twice(getm_min_pos(a, b)), getm_positive_i(lin) ? lin : 0.0);
        break;
    }
    case GETM_SCHEME_MUSCL: pa = getm_min_pos(getm_twice(getm_min_pos(a, b)), getm_half(__dadd_rn(a, b))); break;
    case GETM_SCHEME_P2_PDM:
        if (a == 0.0 || b == 0.0) return 0.0;  // its bounds may be negative beyond Courant numbers of 1
        pa = getm_fmin_i(getm_fmin_i(__dmul_rn(tf.rcoef, b), __fma_rn(tf.lin1, b, __dmul_rn(tf.lin0, a))),
                         __dmul_rn(tf.cap, a));
        break;
    case GETM_SCHEME_SPLMAX13:
        pa = getm_min_pos(getm_twice(getm_min_pos(a, b)),
                          __dmul_rn(1.0 / 3.0, __dadd_rn(__dadd_rn(a, b), getm_max_pos(a, b))));
        break;
    case GETM_SCHEME_SUPERBEE:  // max(min(2b, a), min(b, 2a))
        pa = getm_min_pos(getm_twice(getm_min_pos(a, b)), getm_max_pos(a, b));
        break;
    default: return 0.0;
    }
    return getm_negate_if(pa, hd < 0);
}

__device__ __forceinline__ bool getm_flux_point(int m) { return m == 1 || m == 2; }

// u*u + v*v rounded after each operation (no contraction into an FMA), so
// every kernel that forms a speed from two components gets the same bits.
__device__ __forceinline__ double getm_speed2(double u, double v) { return __dadd_rn(__dmul_rn(u, u), __dmul_rn(v, v)); }
__device__ __forceinline__ float getm_speed2(float u, float v) { return __fadd_rn(__fmul_rn(u, u), __fmul_rn(v, v)); }
