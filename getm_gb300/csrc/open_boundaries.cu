// Open-boundary conditions and mirroring for sm_103a.
//
// Reference: python/pygetm/open_boundaries.py (ZeroGradient :338-356,
// Clamped :358-375, Flather :377-416, Sponge :195-336, mirroring :848-917
// with core.Array.mirror python/pygetm/core.py:723-728) as driven by
// simulation.py:1160-1168 (tracers), :1252-1257 (elevation), :1545-1550
// (depths) and momentum.py:679, :699, :1212 (transports).
//
// A boundary has a few hundred to a few thousand points, so these kernels are
// bound by their launches and a few latencies.  The reference updates its
// boundaries one after the other, and a zero-gradient point next to a corner
// reads a point of another boundary; but no level or tracer looks at another,
// so one block takes a plane (of one level and tracer) through all boundaries
// in the reference's order, with a block barrier between them, and one launch
// does them all (a shelf sea's six boundaries: elevation 6 x 4.7 -> 15 us, eight
// tracers of 20 levels 6 x 20 -> 20 us).  A boundary longer than a block's points
// would go round the block's threads again and again on one SM: it gets a launch
// of its own, its points spread over blocks (ob_launches).
#include <math.h>

#include <algorithm>

#include "getm_common.cuh"

#define OB_THREADS 128
// Most points of a boundary that one block takes with others, and its threads.
// us for six boundaries, one launch each / all in one block per plane (elevation,
// of 256 threads: Flather, clamped; tracers, a thread per point: two clamped,
// two and eight with sponges, 20 levels):
//   240 points   16.9, 10.2; 11.4, 37.9, 116  /  15.9, 5.3; 4.3, 24, 37
//   400 points   16.9, 10.2; 11.6, 40, 127    /  26, 8.4; 4.6, 32, 52
//   1000 points  16.9, 10.2; 11.9, 48, 152    /  56, 15; 6.0, 67, 133
// The elevation is bound by one SM's FP64 pipe (square root and quotient), the
// sponges by its loads and stores.
#define OB_BLOCK 256
#define OB_TRACER_BLOCK 512

namespace {

__device__ __forceinline__ double np_maximum(double lo, double x) { return isnan(x) ? x : fmax(lo, x); }

// The boundaries of a launch, in order: ranges start, stop of the point tables.
struct ObRanges {
    int n;
    int start[GETM_MAX_BOUNDARIES], stop[GETM_MAX_BOUNDARIES];
};

// elevation at the boundary points (open_boundaries.py:338-416), clipped to its
// minimum Dmin - H (simulation.py:580-582); one block for several boundaries
__global__ void __launch_bounds__(OB_BLOCK)
    ob_elevation_kernel(ObRanges r, int nx, const int* bi, const int* bj, const int* type, const int* di,
                        const int* dj, const int* side, const double* sign, const double* H, const double* Dclip,
                        const double* U, const double* V, const double* z_ext, const double* flow_ext, double Dmin,
                        double* z)
{
    for (int b = 0; b < r.n; b++) {
        if (b > 0) __syncthreads();
        for (int p = r.start[b] + blockIdx.x * blockDim.x + threadIdx.x; p < r.stop[b]; p += gridDim.x * blockDim.x) {
            const long long q = (long long)bj[p] * nx + bi[p];
            double v;
            switch (type[p]) {
            case 1:  // ZERO_GRADIENT
                v = z[(long long)(bj[p] + dj[p]) * nx + (bi[p] + di[p])];
                break;
            case 3:  // CLAMPED
                v = z_ext[p];
                break;
            default: {  // FLATHER_ELEV (4), FLATHER_TRANSPORT (-4)
                // transport at the velocity point just inside (extract_uv_in, :149-152)
                double tp;
                switch (side[p]) {
                case 1: tp = U[q]; break;       // WEST: U(j, l)
                case 3: tp = U[q - 1]; break;   // EAST: U(j, l-1)
                case 4: tp = V[q]; break;       // SOUTH: V(l, i)
                default: tp = V[q - nx]; break; // NORTH: V(l-1, i)
                }
                const double D = Dclip[q];
                const double ext = type[p] == 4 ? flow_ext[p] * D : flow_ext[p];
                v = z_ext[p] - sign[p] * (tp - ext) / sqrt(D * GETM_G);
                break;
            }
            }
            z[q] = np_maximum(Dmin - H[q], v);
        }
    }
}

// tracer values at the boundary points for every level (grid x) and tracer (grid
// y; grid z: a single boundary's points) of the batch (ZeroGradient, Clamped; Sponge also relaxes the n points
// inward: v += sp_m (bdy - v), sp_m = ((n - m) / (n + 1))^2, only where the
// mask is 1, open_boundaries.py:235-336 without flow-dependent relaxation)
template <typename T>
struct ObTracerArgs {
    ObRanges r;
    int nx, nz, nsponge;
    long long plane;
    const int *bi, *bj, *type, *di, *dj, *mask;
    int ntracer;
    T* var[16];
    const T* bdy[16];  // (nz, np) prescribed values per tracer
    int np;
};

template <typename T>
__global__ void __launch_bounds__(OB_TRACER_BLOCK) ob_tracer_kernel(const __grid_constant__ ObTracerArgs<T> a)
{
    const int k = blockIdx.x, t = blockIdx.y;
    T* f = a.var[t];
    for (int b = 0; b < a.r.n; b++) {
        if (b > 0) __syncthreads();
        for (int p = a.r.start[b] + blockIdx.z * blockDim.x + threadIdx.x; p < a.r.stop[b]; p += gridDim.z * blockDim.x) {
            const long long q = (long long)a.bj[p] * a.nx + a.bi[p] + k * a.plane;
            const int ty = a.type[p];
            if (ty == 1) {
                f[q] = f[q + (long long)a.dj[p] * a.nx + a.di[p]];
            } else {
                const T bv = a.bdy[t][(long long)k * a.np + p];
                f[q] = bv;
                if (ty == 5) {
                    for (int m = 0; m < a.nsponge; m++) {
                        const long long o = (long long)(m + 1) * ((long long)a.dj[p] * a.nx + a.di[p]);
                        const long long q2 = (long long)a.bj[p] * a.nx + a.bi[p] + o;  // 2D index of the sponge point
                        if (a.mask[q2] != 1) continue;
                        const T r = (T)(a.nsponge - m) / (T)(a.nsponge + 1);
                        f[q + o] = f[q + o] + (r * r) * (bv - f[q + o]);
                    }
                }
            }
        }
    }
}

// core.Array.mirror: field[tgt] = field[src] for n pairs of flat 2D indices
// and nlev levels, with numpy's fancy-assignment semantics (every source is
// read before any target is written: a point can be the target of one pair
// and the source of another): one block per level holds the sources in
// registers over a block barrier, or, with more than MR_BLOCK * MR_HOLD pairs, a
// gather and a scatter launch (us, one level / 40 levels: 1440 pairs 3.1 / 3.7 with
// two launches, 2.8 / 2.9 with one; 2400 pairs 3.1 / 3.9 and 3.8 / 4.0).
constexpr int MR_BLOCK = 512, MR_HOLD = 3;

template <typename T>
__global__ void __launch_bounds__(MR_BLOCK) mirror_kernel(int n, const int* src, const int* tgt, long long plane, T* field)
{
    T* f = field + blockIdx.x * plane;
    T v[MR_HOLD];
#pragma unroll
    for (int m = 0; m < MR_HOLD; m++) {
        const int p = m * MR_BLOCK + threadIdx.x;
        if (p < n) v[m] = f[src[p]];
    }
    __syncthreads();
#pragma unroll
    for (int m = 0; m < MR_HOLD; m++) {
        const int p = m * MR_BLOCK + threadIdx.x;
        if (p < n) f[tgt[p]] = v[m];
    }
}

template <typename T>
__global__ void mirror_gather_kernel(int n, const int* src, int nlev, long long plane, const T* field, T* work)
{
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    const int k = blockIdx.y;
    if (p >= n || k >= nlev) return;
    work[(long long)k * n + p] = field[src[p] + k * plane];
}

template <typename T>
__global__ void mirror_scatter_kernel(int n, const int* tgt, int nlev, long long plane, const T* work, T* field)
{
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    const int k = blockIdx.y;
    if (p >= n || k >= nlev) return;
    field[tgt[p] + k * plane] = work[(long long)k * n + p];
}

// Prescribed elevation from harmonic constituents at model time *time:
// z_p = sum over c of amp_c(p) cos(*time om_c + ph_c(p)), every product and sum
// rounded as written; start: the sum's first constituents (else added to z).
struct ObTide {
    int n;
    double om[GETM_MAX_CONSTITUENTS];
    const double *amp[GETM_MAX_CONSTITUENTS], *ph[GETM_MAX_CONSTITUENTS];
};

__global__ void __launch_bounds__(OB_THREADS) ob_tide_kernel(int np, const __grid_constant__ ObTide t,
                                                             const double* time, double* z, int start)
{
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= np) return;
    const double now = *time;
    double v = start ? 0.0 : z[p];
    for (int c = 0; c < t.n; c++)
        v = __dadd_rn(v, __dmul_rn(t.amp[c][p], cos(__dadd_rn(__dmul_rn(now, t.om[c]), t.ph[c][p]))));
    z[p] = v;
}

// Depths at the velocity points just outside boundaries: z_T_half.mirror(z_U)
// followed by elevation2depth and alpha there (simulation.py:1545-1552)
__global__ void ob_depth_kernel(int n, const int* srcT, const int* tgt, const double* z, const double* zo,
                                const double* Hv, const int* mv, double Dmin, double twoDmin, double ialpha,
                                double* work, double* D, double* alpha)
{
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    const int s = srcT[p], t = tgt[p];
    const double zh = (zo[s] + z[s]) * 0.5;
    work[t] = zh;
    if (mv[t] != 0) {
        const double d = fmax(Hv[t] + zh, Dmin);
        D[t] = d;
        alpha[t] = fmax(0.0, fmin(1.0, (d - twoDmin) * ialpha));
    }
}

}  // namespace

static int ob_ranges(ObRanges& r, int nrange, const int* ranges, int np)
{
    if (nrange < 0 || nrange > GETM_MAX_BOUNDARIES || (nrange && !ranges)) return GETM_ERR_ARG;
    r.n = nrange;
    for (int b = 0; b < nrange; b++) {
        r.start[b] = ranges[2 * b];
        r.stop[b] = ranges[2 * b + 1];
        if (r.start[b] < 0 || r.stop[b] < r.start[b] || r.stop[b] > np) return GETM_ERR_ARG;
    }
    return GETM_OK;
}

// The boundaries in launches, in order: as many at a time as have up to `most`
// points each, a longer one by itself; launch(ranges, points of the longest).
template <typename F>
static int ob_launches(const ObRanges& r, int most, F launch)
{
    auto points = [&](int b) { return r.stop[b] - r.start[b]; };
    for (int b = 0; b < r.n;) {
        ObRanges g;
        g.n = 0;
        int longest = 0;
        do {
            g.start[g.n] = r.start[b];
            g.stop[g.n++] = r.stop[b];
            longest = std::max(longest, points(b));
        } while (++b < r.n && longest <= most && points(b) <= most);
        if (longest == 0) continue;
        const int rc = launch(g, longest);
        if (rc) return rc;
    }
    return GETM_OK;
}

extern "C" int getm_open_boundary_tide(int np, int nconstituent, const double* om, const double* const* amp,
                                       const double* const* phase, const double* time, double* z, cudaStream_t stream)
{
    if (np < 0 || nconstituent < 0 || (nconstituent && (!om || !amp || !phase)) || !time || !z) return GETM_ERR_ARG;
    if (np == 0) return GETM_OK;
    for (int done = 0; done == 0 || done < nconstituent; done += GETM_MAX_CONSTITUENTS) {
        ObTide t;
        t.n = nconstituent - done < GETM_MAX_CONSTITUENTS ? nconstituent - done : GETM_MAX_CONSTITUENTS;
        for (int c = 0; c < t.n; c++) {
            if (!amp[done + c] || !phase[done + c]) return GETM_ERR_ARG;
            t.om[c] = om[done + c];
            t.amp[c] = amp[done + c];
            t.ph[c] = phase[done + c];
        }
        ob_tide_kernel<<<getm_div_up(np, OB_THREADS), OB_THREADS, 0, stream>>>(np, t, time, z, done == 0);
        GETM_CHECK_LAUNCH();
    }
    return GETM_OK;
}

extern "C" int getm_open_boundary_elevations(int nrange, const int* ranges, int np, int nx, const int* i, const int* j,
                                            const int* type, const int* di, const int* dj, const int* side,
                                            const double* inflow_sign, const double* H, const double* Dclip,
                                            const double* U, const double* V, const double* z_ext,
                                            const double* flow_ext, double Dmin, double* z, cudaStream_t stream)
{
    ObRanges r;
    if (nx < 1 || ob_ranges(r, nrange, ranges, np)) return GETM_ERR_ARG;
    if (nrange == 0) return GETM_OK;
    const void* ptrs[] = {i, j, type, di, dj, side, inflow_sign, H, Dclip, U, V, z_ext, flow_ext, z};
    for (const void* q : ptrs)
        if (!q) return GETM_ERR_ARG;
    return ob_launches(r, OB_BLOCK, [&](const ObRanges& g, int longest) {
        const bool alone = longest > OB_BLOCK;
        ob_elevation_kernel<<<alone ? getm_div_up(longest, OB_THREADS) : 1, alone ? OB_THREADS : OB_BLOCK, 0, stream>>>(
            g, nx, i, j, type, di, dj, side, inflow_sign, H, Dclip, U, V, z_ext, flow_ext, Dmin, z);
        GETM_CHECK_LAUNCH();
        return GETM_OK;
    });
}

extern "C" int getm_open_boundary_elevation(int start, int stop, int nx, const int* i, const int* j,
                                            const int* type, const int* di, const int* dj, const int* side,
                                            const double* inflow_sign, const double* H, const double* Dclip,
                                            const double* U, const double* V, const double* z_ext,
                                            const double* flow_ext, double Dmin, double* z, cudaStream_t stream)
{
    if (stop == start && start >= 0 && nx >= 1) return GETM_OK;
    const int range[2] = {start, stop};
    return getm_open_boundary_elevations(1, range, stop, nx, i, j, type, di, dj, side, inflow_sign, H, Dclip, U, V,
                                         z_ext, flow_ext, Dmin, z, stream);
}

template <typename T>
static int ob_tracer_impl(int nrange, const int* ranges, int np, int nx, int ny, int nz, int nsponge, const int* i,
                          const int* j, const int* type, const int* di, const int* dj, const int* mask, int ntracer,
                          T* const* vars, const T* const* bdy, cudaStream_t stream)
{
    ObTracerArgs<T> a;
    if (ob_ranges(a.r, nrange, ranges, np) || nx < 1 || ny < 1 || nz < 1 || nsponge < 0 || ntracer < 0 ||
        ntracer > 16)
        return GETM_ERR_ARG;
    int points = 0;
    for (int b = 0; b < nrange; b++) points += a.r.stop[b] - a.r.start[b];
    if (points == 0 || ntracer == 0) return GETM_OK;
    if (!i || !j || !type || !di || !dj || !mask || !vars || !bdy) return GETM_ERR_ARG;
    a.nx = nx; a.nz = nz; a.nsponge = nsponge; a.np = np;
    a.plane = (long long)nx * ny;
    a.bi = i; a.bj = j; a.type = type; a.di = di; a.dj = dj; a.mask = mask; a.ntracer = ntracer;
    for (int t = 0; t < ntracer; t++) {
        if (!vars[t] || !bdy[t]) return GETM_ERR_ARG;
        a.var[t] = vars[t];
        a.bdy[t] = bdy[t];
    }
    return ob_launches(ObRanges(a.r), OB_TRACER_BLOCK, [&](const ObRanges& g, int longest) {
        a.r = g;
        const bool alone = longest > OB_TRACER_BLOCK;
        const int threads = alone ? OB_BLOCK : std::max(OB_BLOCK, (longest + 31) / 32 * 32);
        ob_tracer_kernel<T><<<dim3(nz, ntracer, alone ? getm_div_up(longest, OB_BLOCK) : 1), threads, 0, stream>>>(a);
        GETM_CHECK_LAUNCH();
        return GETM_OK;
    });
}

extern "C" int getm_open_boundary_tracers(int start, int stop, int np, int nx, int ny, int nz, int nsponge,
                                          const int* i, const int* j, const int* type, const int* di,
                                          const int* dj, const int* mask, int ntracer, double* const* vars,
                                          const double* const* bdy, cudaStream_t stream)
{
    const int range[2] = {start, stop};
    return ob_tracer_impl<double>(1, range, np, nx, ny, nz, nsponge, i, j, type, di, dj, mask, ntracer, vars, bdy,
                                  stream);
}

extern "C" int getm_open_boundary_tracers_f32(int start, int stop, int np, int nx, int ny, int nz, int nsponge,
                                              const int* i, const int* j, const int* type, const int* di,
                                              const int* dj, const int* mask, int ntracer, float* const* vars,
                                              const float* const* bdy, cudaStream_t stream)
{
    const int range[2] = {start, stop};
    return ob_tracer_impl<float>(1, range, np, nx, ny, nz, nsponge, i, j, type, di, dj, mask, ntracer, vars, bdy,
                                 stream);
}

// every boundary in turn, one launch
extern "C" int getm_open_boundaries_tracers(int nrange, const int* ranges, int np, int nx, int ny, int nz,
                                            int nsponge, const int* i, const int* j, const int* type, const int* di,
                                            const int* dj, const int* mask, int ntracer, double* const* vars,
                                            const double* const* bdy, cudaStream_t stream)
{
    return ob_tracer_impl<double>(nrange, ranges, np, nx, ny, nz, nsponge, i, j, type, di, dj, mask, ntracer, vars,
                                  bdy, stream);
}

extern "C" int getm_open_boundaries_tracers_f32(int nrange, const int* ranges, int np, int nx, int ny, int nz,
                                                int nsponge, const int* i, const int* j, const int* type,
                                                const int* di, const int* dj, const int* mask, int ntracer,
                                                float* const* vars, const float* const* bdy, cudaStream_t stream)
{
    return ob_tracer_impl<float>(nrange, ranges, np, nx, ny, nz, nsponge, i, j, type, di, dj, mask, ntracer, vars,
                                 bdy, stream);
}

template <typename T>
static int mirror_impl(int n, const int* src, const int* tgt, int nlev, long long plane, T* field, T* work,
                       cudaStream_t stream)
{
    if (n < 0 || nlev < 1 || plane < 1) return GETM_ERR_ARG;
    if (n == 0) return GETM_OK;
    if (!src || !tgt || !field || !work) return GETM_ERR_ARG;
    if (n <= MR_BLOCK * MR_HOLD) {
        mirror_kernel<T><<<nlev, MR_BLOCK, 0, stream>>>(n, src, tgt, plane, field);
        GETM_CHECK_LAUNCH();
        return GETM_OK;
    }
    dim3 grid(getm_div_up(n, OB_THREADS), nlev);
    mirror_gather_kernel<T><<<grid, OB_THREADS, 0, stream>>>(n, src, nlev, plane, field, work);
    GETM_CHECK_LAUNCH();
    mirror_scatter_kernel<T><<<grid, OB_THREADS, 0, stream>>>(n, tgt, nlev, plane, work, field);
    GETM_CHECK_LAUNCH();
    return GETM_OK;
}

extern "C" int getm_mirror(int n, const int* src, const int* tgt, int nlev, long long plane, double* field,
                           double* work, cudaStream_t stream)
{
    return mirror_impl<double>(n, src, tgt, nlev, plane, field, work, stream);
}

extern "C" int getm_mirror_f32(int n, const int* src, const int* tgt, int nlev, long long plane, float* field,
                               float* work, cudaStream_t stream)
{
    return mirror_impl<float>(n, src, tgt, nlev, plane, field, work, stream);
}

extern "C" int getm_open_boundary_depth(int n, const int* srcT, const int* tgt, const double* z, const double* zo,
                                        const double* H, const int* mask, double Dmin, double Dcrit, double* work,
                                        double* D, double* alpha, cudaStream_t stream)
{
    if (n < 0) return GETM_ERR_ARG;
    if (n == 0) return GETM_OK;
    if (!srcT || !tgt || !z || !zo || !H || !mask || !work || !D || !alpha) return GETM_ERR_ARG;
    ob_depth_kernel<<<getm_div_up(n, OB_THREADS), OB_THREADS, 0, stream>>>(
        n, srcT, tgt, z, zo, H, mask, Dmin, 2 * Dmin, 1.0 / (Dcrit - 2 * Dmin), work, D, alpha);
    GETM_CHECK_LAUNCH();
    return GETM_OK;
}
