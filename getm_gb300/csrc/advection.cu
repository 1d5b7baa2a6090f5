// TVD directional-split advection (pygetm.operators.Advection) for sm_103a.
//
// Reference: src/operators/advection_schemes/advection.F90.template (u2d :23-121,
// v2d :123-221, w3d :223-374), limiters.h, python/src/wrapper.F90:188-273 and
// the split sequencing of python/pygetm/operators.py:52-193.
//
// GB300 design
// * Horizontal passes are one kernel per direction and stage, batched over all
//   tracers: the face geometry (mask, transport QU, Courant number, upwind
//   side) and the layer-thickness update are computed once per cell and
//   reused for every tracer.  Memory traffic per pass is the algorithmic
//   minimum: read u, hu, h, var; write h, var.
// * The reference updates var and h in place after computing all face fluxes
//   of a layer.  A GPU block cannot see its neighbours' updates in order, so
//   each pass reads from one buffer and writes a complete copy to another
//   (ping-pong through handle-owned work buffers); the stage sequence is laid
//   out so the final stage lands in the caller's arrays.
// * x-direction: a warp covers 31 consecutive cells of a row (32 faces); each
//   face is evaluated once and reaches its second cell by a shuffle.
// * y-direction: blocks of 32 x 16 threads cover 15 rows with the faces
//   exchanged through shared memory, or (float arithmetic, several layers)
//   warps march north with the rows in registers.
// * Vertical pass: a warp's lanes are 32 water columns; each thread sweeps k
//   with a register window, the whole column or (few columns) a segment of it.
//   The per-column update is in place, as in the reference.  The adaptive
//   sub-stepping (itersmax = 200, restart semantics of template :286-368) runs
//   through handle-owned column work arrays.
#include <stdlib.h>
#include <string.h>

#include <cuda_pipeline.h>

#include "advection_passes.cuh"


// ---------------------------------------------------------------------------
// grid handles
// ---------------------------------------------------------------------------
extern "C" int getm_create_grid(int imin, int imax, int jmin, int jmax, int kmin, int kmax,
                                int halox, int haloy, getm_grid** grid)
{
    if (!grid || imax < imin || jmax < jmin || kmax < kmin - 1 || halox < 0 || haloy < 0)
        return GETM_ERR_ARG;
    getm_grid* g = (getm_grid*)calloc(1, sizeof(getm_grid));
    if (!g) return GETM_ERR_ALLOC;
    g->imin = imin; g->imax = imax; g->jmin = jmin; g->jmax = jmax;
    g->kmin = kmin; g->kmax = kmax; g->halox = halox; g->haloy = haloy;
    g->nx_ = imax - imin + 1 + 2 * halox;
    g->ny_ = jmax - jmin + 1 + 2 * haloy;
    *grid = g;
    return GETM_OK;
}

extern "C" int getm_grid_finalize(getm_grid* grid)
{
    if (grid) {
        cudaFree(grid->dx_f); cudaFree(grid->dy_f); cudaFree(grid->idx_f);
        cudaFree(grid->idy_f); cudaFree(grid->iarea_f);
    }
    free(grid);
    return GETM_OK;
}

__global__ void to_float_kernel(long long n, const double* src, float* dst)
{
    long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (p < n) dst[p] = (float)src[p];
}

// The float copies of a grid's metrics, converted on `stream` after every
// earlier write of the metrics on that stream, and complete on return (the
// wait is for `stream` only).
static int grid_float_metrics_on(getm_grid* g, cudaStream_t stream)
{
    const long long n = (long long)g->nx_ * g->ny_;
    const double* src[5] = {g->dx, g->dy, g->idx, g->idy, g->iarea};
    float** dst[5] = {&g->dx_f, &g->dy_f, &g->idx_f, &g->idy_f, &g->iarea_f};
    for (int q = 0; q < 5; q++) {
        if (!src[q]) continue;  // metric not registered on this grid
        float* d = NULL;
        if (cudaMalloc(&d, n * sizeof(float)) != cudaSuccess) return GETM_ERR_ALLOC;
        to_float_kernel<<<getm_div_up(n, 256), 256, 0, stream>>>(n, src[q], d);
        GETM_CHECK_LAUNCH();
        *dst[q] = d;
    }
    if (!g->iarea_f) {  // grids without cell areas (velocity grids): mark as built
        if (cudaMalloc(&g->iarea_f, sizeof(float)) != cudaSuccess) return GETM_ERR_ALLOC;
    }
    if (cudaStreamSynchronize(stream) != cudaSuccess) return GETM_ERR_CUDA;
    return GETM_OK;
}

// First use by a float kernel of a grid whose copies were not made with
// getm_grid_float_metrics: the metrics may have been written on any stream,
// so the conversion is ordered after all work on the device.
int getm_grid_f32_metrics(getm_grid* g, cudaStream_t stream)
{
    if (!g) return GETM_ERR_ARG;
    if (g->iarea_f) return GETM_OK;  // built last: its presence means all are there
    if (cudaDeviceSynchronize() != cudaSuccess) return GETM_ERR_CUDA;
    return grid_float_metrics_on(g, stream);
}

extern "C" int getm_grid_float_metrics(getm_grid* g, cudaStream_t stream)
{
    if (!g) return GETM_ERR_ARG;
    if (g->iarea_f) return GETM_OK;
    return grid_float_metrics_on(g, stream);
}

extern "C" int getm_grid_set_array(getm_grid* g, const char* name, void* p)
{
    if (!g || !name) return GETM_ERR_ARG;
    if (!strcmp(name, "mask")) g->mask = (const int*)p;
    else if (!strcmp(name, "dx")) g->dx = (const double*)p;
    else if (!strcmp(name, "dy")) g->dy = (const double*)p;
    else if (!strcmp(name, "idx")) g->idx = (const double*)p;
    else if (!strcmp(name, "idy")) g->idy = (const double*)p;
    else if (!strcmp(name, "iarea")) g->iarea = (const double*)p;
    else if (!strcmp(name, "area")) g->area = (const double*)p;
    else return GETM_ERR_ARG;
    return GETM_OK;
}

// ---------------------------------------------------------------------------
// advection handle: scheme plus device work buffers (grown on demand)
// ---------------------------------------------------------------------------
struct getm_advection {
    int scheme;
    getm_grid* tgrid;
    size_t n3;                 // elements of one 3D field the buffers are sized for
    double* hbuf[2];           // layer-thickness ping-pong buffers
    double* colbuf[2];         // vertical sub-stepping work arrays (haux: n3, faux: 2 n3 doubles)
    double* tmp[GETM_MAX_BATCH * 8];  // per-tracer ping-pong buffers
    int ntmp;
    int* status;               // device status word (GETM_ERR_ITERS)
};

static void adv_free_buffers(getm_advection* a)
{
    // (cudaFree waits for the whole device: never called without a buffer)
    for (int i = 0; i < 2; i++) if (a->hbuf[i]) { cudaFree(a->hbuf[i]); a->hbuf[i] = NULL; }
    for (int i = 0; i < 2; i++) if (a->colbuf[i]) { cudaFree(a->colbuf[i]); a->colbuf[i] = NULL; }
    for (int i = 0; i < a->ntmp; i++) if (a->tmp[i]) { cudaFree(a->tmp[i]); a->tmp[i] = NULL; }
    a->ntmp = 0;
    a->n3 = 0;
}

// Make sure the work buffers can hold 3D fields of n3 elements and ntracer
// per-tracer ping-pong copies.  Allocation happens on first use only (so a
// warm-up call before stream capture makes later calls capturable).
static int adv_reserve(getm_advection* a, size_t n3, int ntracer)
{
    if (ntracer > GETM_MAX_BATCH * 8) return GETM_ERR_ARG;
    if (n3 > a->n3) {
        adv_free_buffers(a);
        for (int i = 0; i < 2; i++)
            if (cudaMalloc(&a->hbuf[i], n3 * sizeof(double)) != cudaSuccess) return GETM_ERR_ALLOC;
        // colbuf[1] holds the intermediate sub-steps of a pair of fields
        // stepped together by the w pass (two fields of up to 8 bytes)
        if (cudaMalloc(&a->colbuf[0], n3 * sizeof(double)) != cudaSuccess) return GETM_ERR_ALLOC;
        if (cudaMalloc(&a->colbuf[1], 2 * n3 * sizeof(double)) != cudaSuccess) return GETM_ERR_ALLOC;
        a->n3 = n3;
    }
    while (a->ntmp < ntracer) {
        if (cudaMalloc(&a->tmp[a->ntmp], a->n3 * sizeof(double)) != cudaSuccess) return GETM_ERR_ALLOC;
        a->ntmp++;
    }
    return GETM_OK;
}

extern "C" int getm_advection_create(int scheme, getm_grid* tgrid, getm_advection** out)
{
    if (!out || scheme < GETM_SCHEME_HSIMT || scheme > GETM_SCHEME_UPSTREAM) return GETM_ERR_ARG;
    getm_advection* a = (getm_advection*)calloc(1, sizeof(getm_advection));
    if (!a) return GETM_ERR_ALLOC;
    a->scheme = scheme;
    a->tgrid = tgrid;
    if (cudaMalloc(&a->status, sizeof(int)) != cudaSuccess) { free(a); return GETM_ERR_ALLOC; }
    cudaMemset(a->status, 0, sizeof(int));
    *out = a;
    return GETM_OK;
}

extern "C" int getm_advection_finalize(getm_advection* a)
{
    if (!a) return GETM_OK;
    adv_free_buffers(a);
    cudaFree(a->status);
    free(a);
    return GETM_OK;
}

extern "C" int getm_advection_get_status(getm_advection* a, cudaStream_t stream)
{
    if (!a) return GETM_ERR_ARG;
    int h = 0;
    if (cudaMemcpyAsync(&h, a->status, sizeof(int), cudaMemcpyDeviceToHost, stream) != cudaSuccess) return GETM_ERR_CUDA;
    if (cudaStreamSynchronize(stream) != cudaSuccess) return GETM_ERR_CUDA;
    return h;
}

// ---- kernels (one pass per launch) ------------------------------------------
// grid (segments, ceil(ny_ / 8), nk): warp (ty) of block (x, y, k) owns row j = 8 y + ty of layer k
template <typename S, typename V, typename C>
__global__ void __launch_bounds__(256) hpass_x_inc_kernel(HPassArgs<S, V> a)
{
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    if (j >= a.ny_) return;  // whole warp
    hpass_x_inc_rows<S, 1, NoEpi, V, C>(a, blockIdx.x, j, blockIdx.z, threadIdx.x);
}

// grid (pairs of fields, y, nk): each warp of block (g, y, k) sweeps nrow rows of layer k
template <typename S, typename V = S>
__global__ void __launch_bounds__(256) hpass_x_vec_kernel(HPassArgs<S, V> a, int nrow)
{
    const int j0 = (blockIdx.y * blockDim.y + threadIdx.y) * nrow;
    if (j0 >= a.ny_) return;  // whole warp
    hpass_x_vec_rows<S, V>(a, j0, min(nrow, a.ny_ - j0), blockIdx.z, threadIdx.x, 2 * blockIdx.x);
}

// The four-cells-per-lane x pass applies: rows of whole 16-byte vectors and
// every pointer it reads or writes 16-byte aligned.
template <typename S, typename V>
static bool xpass_vec_ok(const HPassArgs<S, V>& a)
{
    if (a.nk < 2 || a.nx_ % 4 != 0 || a.ntracer > GETM_MAX_BATCH) return false;
    auto al = [](const void* p) { return ((uintptr_t)p & 15u) == 0; };
    if (!al(a.umask) || !al(a.tmask) || !al(a.dy_f) || !al(a.idx_f) || !al(a.iA_f) || !al(a.u) || !al(a.hu) ||
        !al(a.h_in) || !al(a.h_out) || (a.Ah && !al(a.Ah)))
        return false;
    for (int t = 0; t < a.ntracer; t++)
        if (!al(a.fin[t]) || !al(a.fout[t])) return false;
    return true;
}

template <typename S, typename V, typename C, int BY>
__global__ void __launch_bounds__(32 * BY) hpass_y_inc_kernel(HPassArgs<S, V> a)
{
    __shared__ YIncSmem<S, C, BY> sm;
    hpass_y_inc_body<S, NoEpi, V, C, BY>(a, blockIdx.x, blockIdx.y, blockIdx.z, threadIdx.x, threadIdx.y, sm);
}

template <typename S, int NT, typename V = S>
__global__ void __launch_bounds__(256) hpass_y_march_kernel(HPassArgs<S, V> a, int nchunk)
{
    const int w = blockIdx.y * blockDim.y + threadIdx.y;
    const int chunk = w % nchunk, k = w / nchunk;
    if (k >= a.nk) return;  // whole warp
    // a group of NT tracers per block z; with no tracers one sweep updates h
    hpass_y_march_body<S, NT, V>(a, blockIdx.x, chunk, k, threadIdx.x, NT * blockIdx.z);
}

// Launch one horizontal pass (storage type S, velocity type V, arithmetic C).
template <typename S, typename V, typename C>
static int launch_hpass_c(int direction, HPassArgs<S, V>& a, cudaStream_t stream)
{
    constexpr bool f64 = std::is_same<C, double>::value;
    if (direction == 1) {
        const int rows = getm_tune(GETM_TUNE_XPASS_ROWS);
        dim3 block(32, rows);
        bool vec = false;
        // four cells per lane: float arithmetic only.  The FP64 form is bound
        // by its FP64 instructions, and the one-cell kernel forms a face's
        // geometry once for all fields where the sweep repeats it per pair
        if constexpr (!f64) vec = getm_tune(GETM_TUNE_XPASS_VEC) && xpass_vec_ok(a);
        if (vec) {
            // rows per warp: four where that fills the chunks better (a 404-cell
            // row by itself fills 3.2 of its four, a 244-cell row 1.9 of two) and
            // leaves 16 warps per SM; at most two warps per block, so that the
            // last wave of blocks is short.  us per five-pass split of 240 x 200 x
            // 20 with eight fields: pairs one after the other 578, side by side
            // 566, and one row per warp 502
            const int npair = a.ntracer > 0 ? (a.ntracer + 1) / 2 : 1, nq = a.nx_ / 4;
            auto chunks = [&](int n) { return getm_div_up((long long)n * nq, 32) * (4 / n); };  // of four rows
            int nrow = 4;
            while (nrow > 1 && (chunks(nrow / 2) * 97 <= chunks(4) * 100 ||
                                (long long)getm_div_up(a.ny_, nrow) * a.nk * npair < 16 * GETM_SMS))
                nrow /= 2;
            block.y = rows < 2 || getm_div_up(a.ny_, 2 * nrow) > 65535 ? rows : 2;  // (a grid's most blocks)
            dim3 grid(npair, getm_div_up(getm_div_up(a.ny_, nrow), block.y), a.nk);
            if constexpr (!f64) hpass_x_vec_kernel<S, V><<<grid, block, 0, stream>>>(a, nrow);
        } else {
            // lane 0 of the first segment handles the face west of cell 0
            dim3 grid(getm_div_up(a.nx_ + 1, HX_STRIDE), getm_div_up(a.ny_, rows), a.nk);
            hpass_x_inc_kernel<S, V, C><<<grid, block, 0, stream>>>(a);
        }
    } else if (f64 || a.nk < 4) {
        // a single plane: too few columns x layers for marching warps to fill
        // the GPU, so blocks of 32 columns cover tiles instead.  FP64
        // form: the tile kernel forms a face's geometry once for all fields
        // and has a block per 15 rows or less, where the marching kernel repeats the
        // geometry per pair and had blocks for 90 of 152 SMs on 173 x 131 x 23
        const int by = hpass_y_rows((long long)getm_div_up(a.nx_, 32) * a.nk, a.ny_, f64);
        const dim3 block(32, by), grid(getm_div_up(a.nx_, 32), getm_div_up(a.ny_ + 1, by - 1), a.nk);
        if (by == 16) hpass_y_inc_kernel<S, V, C, 16><<<grid, block, 0, stream>>>(a);
        else hpass_y_inc_kernel<S, V, C, 4><<<grid, block, 0, stream>>>(a);
    } else {
        // rows a warp marches: the knob's, halved (to four at least, which
        // repeats one face in four) until there are 64 warps per SM: a warp's
        // march is a chain of load latencies.  us per five-pass split with the
        // knob's 32 -> this, groups of fields one after the other -> side by
        // side: 92 x 92 x 20 two FP64-stored fields 140 -> 64, a float field 78 ->
        // 45; 150 x 120 x 30 three 195 -> 151; 240 x 200 x 20 eight 860 -> 578, a float
        // field 120 -> 102; 400 x 300 x 40 two 622 -> 582 (eight rows 594)
        const int nt = a.ntracer >= 2 ? 2 : 1, ngroup = a.ntracer > nt ? getm_div_up(a.ntracer, nt) : 1;
        const long long strips = (long long)getm_div_up(a.nx_, 32) * a.nk * ngroup;
        a.ych = getm_tune(GETM_TUNE_YMARCH_CHUNK);
        while (a.ych > 4 && strips * getm_div_up(a.ny_, a.ych) < 64 * GETM_SMS) a.ych /= 2;
        const int nchunk = getm_div_up(a.ny_, a.ych);
        dim3 block(32, 8);
        dim3 grid(getm_div_up(a.nx_, 32), getm_div_up((long long)nchunk * a.nk, 8), ngroup);
        if constexpr (!f64) {
            if (a.ntracer >= 2) hpass_y_march_kernel<S, 2, V><<<grid, block, 0, stream>>>(a, nchunk);
            else hpass_y_march_kernel<S, 1, V><<<grid, block, 0, stream>>>(a, nchunk);
        }
    }
    GETM_CHECK_LAUNCH();
    return GETM_OK;
}

template <typename T, typename V = T>
static int launch_hpass(int direction, HPassArgs<T, V>& a, cudaStream_t stream)
{
    if constexpr (getm_increment_form<T> || !std::is_same<T, V>::value) {
        return launch_hpass_c<T, V, float>(direction, a, stream);
    } else {
        if (a.increment) return launch_hpass_c<T, V, float>(direction, a, stream);
        return launch_hpass_c<T, V, double>(direction, a, stream);
    }
}

// Fill the direction-dependent fields of HPassArgs from the grid handles
// (wrapper.F90:240-253: direction 1 passes ugrid mask/idx/dy, 2 passes vgrid
// mask/dx/idy).
template <typename T, typename V = T>
static int hpass_setup(HPassArgs<T, V>& a, int direction, const getm_advection* adv, const getm_grid* tg,
                       const getm_grid* vg, int nk, const V* u, const double* Ah, double dt, const double* hu,
                       int increment = 0)
{
    if (!tg || !vg || !u || !hu) return GETM_ERR_ARG;
    if (tg->halox < 2 || tg->haloy < 2) return GETM_ERR_ARG;
    if (!tg->mask || !tg->iarea || !vg->mask) return GETM_ERR_ARG;
    memset(&a, 0, sizeof(a));
    a.nx_ = tg->nx_; a.ny_ = tg->ny_; a.nk = nk;
    a.plane = (long long)tg->nx_ * tg->ny_;
    a.ilo = tg->halox; a.ihi = tg->halox + (tg->imax - tg->imin);
    a.jlo = tg->haloy; a.jhi = tg->haloy + (tg->jmax - tg->jmin);
    a.umask = vg->mask;
    if (direction == 1) { a.idx = vg->idx; a.dy = vg->dy; }
    else { a.idx = vg->idy; a.dy = vg->dx; }
    if (!a.idx || !a.dy) return GETM_ERR_ARG;
    a.tmask = tg->mask; a.iA = tg->iarea; a.Ah = Ah; a.u = u; a.hu = hu; a.dt = dt;
    a.scheme = adv->scheme;
    a.dtf = (float)dt;
    if (getm_increment_form<T> || !std::is_same<T, V>::value || increment) {
        a.increment = 1;
        int rc = getm_grid_f32_metrics(const_cast<getm_grid*>(tg), 0);
        if (!rc) rc = getm_grid_f32_metrics(const_cast<getm_grid*>(vg), 0);
        if (rc) return rc;
        a.iA_f = tg->iarea_f;
        if (direction == 1) { a.idx_f = vg->idx_f; a.dy_f = vg->dy_f; }
        else { a.idx_f = vg->idy_f; a.dy_f = vg->dx_f; }
        if (!a.iA_f || !a.idx_f || !a.dy_f) return GETM_ERR_ARG;
    }
    return GETM_OK;
}

// Run one horizontal stage for ntracer tracers, chunked by GETM_MAX_BATCH.
template <typename T, typename V = T>
static int run_hstage(HPassArgs<T, V>& a, int direction, const double* h_in, double* h_out, int ntracer,
                      const T* const* fin, T* const* fout, cudaStream_t stream)
{
    a.h_in = h_in; a.h_out = h_out;
    int done = 0;
    do {
        int n = ntracer - done;
        if (n > GETM_MAX_BATCH) n = GETM_MAX_BATCH;
        a.ntracer = n;
        for (int t = 0; t < n; t++) { a.fin[t] = fin[done + t]; a.fout[t] = fout[done + t]; }
        int rc = launch_hpass<T, V>(direction, a, stream);
        if (rc) return rc;
        done += n;
    } while (done < ntracer);
    return GETM_OK;
}

// ---------------------------------------------------------------------------
// vertical pass (template w3d :223-374)
// ---------------------------------------------------------------------------
// T: the advected fields; V: w and w_var (T unless given).  T = double, V =
// float is the mixed form with FP64 tracer storage (increment form).
template <typename T, typename V = T>
struct WPassArgs {
    int nx_, ny_, nz;
    long long plane;
    int ilo, ihi, jlo, jhi;
    const int* tmask;
    const V* w;                 // nz+1 levels
    const double* h_in;         // layer thickness at stage start (not modified)
    double* h_out;              // layer thickness after the pass (last tracer's)
    double* haux;               // column work arrays for sub-stepping (nz levels)
    T* faux;
    double dt;
    int scheme;
    int ntracer;
    int* status;
    const V* wvar[GETM_MAX_BATCH];
    T* f[GETM_MAX_BATCH];       // updated in place
};

// The pass is explicit: every level's new value depends only on old values of
// the levels around it.  So on domains with few columns (w_segments) a
// column's levels are shared by several warps, each sweeping a segment k0 ..
// k1-1 upwards; a segment's sweep runs in place: it reads its own levels before
// it overwrites them, and the values of its neighbours' levels that it needs
// (WHalo) are read before a block barrier, after which all segments write.
//
// One sub-step is in increment form (see hpass_x_inc_rows).  With flux_k =
// W_k f + e_k at the interface above level k (W_k = w_var there, 0 at the
// surface) and dh = dtk (w_k - w_{k-1}), the reference update equals
//     f + dtk ((w_k - W_k - w_{k-1} + W_{k-1}) f - e_k + e'_{k-1}) / hn
// with e_k = W_k (face_k - f_k) and e'_{k-1} = W_{k-1} (face_{k-1} - f_k).
// The Courant number |w_var| dt / min(h) * itersm1 equals cfls(k)*itersm1 of
// the reference (cfls = |w_var| dt / min(haux), haux = the sub-step's start
// thickness).  NT fields advected with the same w_var share every thickness
// and velocity load and the face constants; each field keeps its own window.
// V: the velocities and the arithmetic, float (mixed form) or double.  The
// FP64 form takes 13 FP64 instructions per level and 6 per field and level
// (superbee, w_var = w) where the reference's order of evaluation, with its
// five divisions, took about 140.  One thread per column in that order took
// 134 us on 120 x 100 x 30 with one field and 672 us on 173 x 131 x 23 with six
// (HSIMT); this form takes 41 us and 199 us.
//
// The operands of the levels a sweep will need are staged W_STAGE levels
// ahead into a per-thread ring in shared memory by asynchronous copies
// (cp.async): the loads of W_STAGE levels are in flight without holding
// registers.  Each thread reads back only the slots it filled, so no block
// barrier is involved; a slot is refilled only after its level was read.
constexpr int W_STAGE = 6;
constexpr int W_RING = W_STAGE + 1;
constexpr int W_MAXSEG = 8;

// With SEG the two slots after the ring hold the old values of the two levels
// above the segment.
template <bool SEG>
constexpr int w_slots = SEG ? W_RING + 2 : W_RING;

// A warp's ring in the block's dynamic shared memory: h, f, w_var and w of its
// 32 columns, one behind the other at fixed offsets (widest types first, so
// every slot is naturally aligned; one pointer for all four).
extern __shared__ __align__(16) unsigned char w_smem[];

template <bool SEG, typename S, typename V>
struct WRing {
    static_assert(sizeof(S) == 8 || sizeof(S) == sizeof(V), "fields in double or in the velocities' type");
    static constexpr size_t OFF_F = (size_t)w_slots<SEG> * 32 * sizeof(double);
    static constexpr size_t OFF_W = OFF_F + (size_t)w_slots<SEG> * 64 * sizeof(S);
    static constexpr size_t OFF_w = OFF_W + (size_t)W_RING * 32 * sizeof(V);
    static constexpr size_t BYTES = OFF_w + (size_t)W_RING * 32 * sizeof(V);
    int o8, oV;  // the lane's byte offsets of h and of w_var
    __device__ __forceinline__ WRing(int warp, int lane)
        : o8(warp * (int)BYTES + lane * 8), oV(warp * (int)BYTES + (int)OFF_W + lane * (int)sizeof(V))
    {
    }
    __device__ __forceinline__ double& h(int slot) const { return *reinterpret_cast<double*>(w_smem + o8 + slot * 256); }
    __device__ __forceinline__ S& f(int slot, int q) const
    {
        constexpr int n = sizeof(S);
        const int o = n == 8 ? o8 : oV - (int)(OFF_W - OFF_F);  // (V is as wide as a narrow S)
        return *reinterpret_cast<S*>(w_smem + o + (n == 8 ? (int)OFF_F : 0) + (slot * 2 + q) * 32 * n);
    }
    __device__ __forceinline__ V& W(int slot) const
    {
        return *reinterpret_cast<V*>(w_smem + oV + slot * 32 * (int)sizeof(V));
    }
    __device__ __forceinline__ V& w(int slot) const
    {
        return *reinterpret_cast<V*>(w_smem + oV + (int)(OFF_w - OFF_W) + slot * 32 * (int)sizeof(V));
    }
};

// Old values beside a segment, zero where the column ends: levels k0-2 and
// k0-1; those of levels k1 and k1+1 go to the thread's two slots after the ring.
template <int NT, typename S>
struct WHalo {
    S lo2[NT], lo1[NT];
    double hlo;
};

template <int NT, typename S, typename V>
__device__ __forceinline__ WHalo<NT, S> w_halo(long long c, long long P, int nz, int k0, int k1, const double* hs,
                                               const S* const (&fs)[NT], const WRing<true, S, V>& ring)
{
    WHalo<NT, S> H;
#pragma unroll
    for (int q = 0; q < NT; q++) {
        H.lo2[q] = k0 >= 2 ? fs[q][c + (k0 - 2) * P] : S(0);
        H.lo1[q] = k0 >= 1 ? fs[q][c + (k0 - 1) * P] : S(0);
        ring.f(W_RING, q) = k1 < nz ? fs[q][c + k1 * P] : S(0);
        ring.f(W_RING + 1, q) = k1 + 1 < nz ? fs[q][c + (k1 + 1) * P] : S(0);
    }
    H.hlo = k0 >= 1 ? hs[c + (k0 - 1) * P] : 0.0;
    ring.h(W_RING) = k1 < nz ? hs[c + k1 * P] : 0.0;
    ring.h(W_RING + 1) = 0.0;  // (beyond the last interface: not used)
    return H;
}

// e_k and e'_k of the interface between two levels of thickness h0 (below)
// and h1, per field: tf and W are the interface's, d the difference across it,
// dprev and dnext those below and above
__device__ __forceinline__ void w_face(const TvdFace<float>& tf, float W, float dprev, float d, float dnext, float& el,
                                       float& er)
{
    // the limiter is odd: one evaluation for both flow directions
    const bool up = W > 0.f;
    const float lim = getm_tvd_dev_c(tf, d, up ? dprev : dnext);
    const float dev = up ? lim : -lim;
    const float a = __fadd_rn(dev, up ? -d : d);
    el = __fmul_rn(W, up ? dev : a);
    er = __fmul_rn(W, up ? a : dev);
}

__device__ __forceinline__ void w_face(const TvdFace<double>& tf, double W, double dprev, double d, double dnext,
                                       double& el, double& er)
{
    hx_face(tf, getm_positive_i(W), true, W, dprev, d, dnext, 0.0, false, el, er);
}

__device__ __forceinline__ TvdFace<float> w_tvd(int scheme, float W, float dt, float itersm1, float h0, float h1)
{
    const float cfl = __fmul_rn(fabsf(W) * dt / fminf(h0, h1), itersm1);
    return getm_tvd_face_c(scheme, cfl);
}

__device__ __forceinline__ TvdFace<double> w_tvd(int scheme, double W, double dt, double itersm1, double h0, double h1)
{
    const double cfl = __dmul_rn(__dmul_rn(fabs(W), __dmul_rn(dt, itersm1)), getm_rcp(getm_fmin_i(h0, h1)));
    return hx_tvd(scheme, cfl, W);
}

// SEG: the column is split (else k0 = 0, k1 = nz, and nothing lies beside it).
template <int NT, bool SEG, typename S, typename V>
__device__ void w_substep(const WPassArgs<S, V>& a, long long c, int kbeg, int kend, const V* wv, const double* hs,
                          const S* const (&fs)[NT], double* hd, S* const (&fdst)[NT], double dtk, double itersm1,
                          const WHalo<NT, S>& H, const WRing<SEG, S, V>& ring)
{
    const long long P = a.plane;
    const int nz = a.nz;
    const int k0 = SEG ? kbeg : 0, k1 = SEG ? kend : nz;
    const V dtkf = (V)dtk, itf = (V)itersm1, dtf = (V)a.dt;
    const bool own_w = wv == a.w;
    // the differences f[k+1] - f[k] (dk) and f[k] - f[k-1] (dkm1), narrowed:
    // each is formed once, as the level above's is needed next (the
    // downwind-side difference f[k+1] - f[k+2] is -(f[k+2] - f[k+1]), the
    // same bits up to the sign of a zero, which the limiter ignores)
    S fk[NT], fk1[NT];
    V dk[NT], dkm1[NT];
    V erm[NT];  // e'_{k-1}, interface below, deviation from level k
    const long long c0 = c + k0 * P;
    double hk = hs[c0], hk1 = k0 + 1 < k1 ? hs[c0 + P] : (SEG ? ring.h(W_RING) : 0.0);
#pragma unroll
    for (int q = 0; q < NT; q++) {
        fk[q] = fs[q][c0];
        fk1[q] = k0 + 1 < k1 ? fs[q][c0 + P] : (SEG ? ring.f(W_RING, q) : S(0));
        dk[q] = k0 + 1 < nz ? hx_c<V>(fk1[q] - fk[q]) : V(0);
        dkm1[q] = k0 > 0 ? hx_c<V>(fk[q] - H.lo1[q]) : V(0);
        erm[q] = V(0);
    }
    V hkf = hx_c<V>(hk), hk1f = hx_c<V>(hk1);
    V Wm = k0 > 0 ? wv[c0] : V(0);  // W_{k-1} (0 below the bottom level)
    V wkm1 = a.w[c0];
    // the interface values above level k, one level ahead
    V Wn = k0 < nz - 1 ? wv[c0 + P] : V(0);
    V wkn = a.w[c0 + P];
    // level L's operands (at offset o) into a slot: those of the segment's own
    // levels, and the velocities of the column; one commit group per level
    auto stage = [&](int L, long long o, int slot) {
        if (L < k1) {
#pragma unroll
            for (int q = 0; q < NT; q++) __pipeline_memcpy_async(&ring.f(slot, q), &fs[q][o], sizeof(S));
            __pipeline_memcpy_async(&ring.h(slot), &hs[o], sizeof(double));
        }
        if (L <= k1 && L < nz) __pipeline_memcpy_async(&ring.W(slot), &wv[o], sizeof(V));
        if (L <= k1) __pipeline_memcpy_async(&ring.w(slot), &a.w[o], sizeof(V));
        __pipeline_commit();
    };
#pragma unroll 1
    for (int n = 0; n < W_STAGE; n++) stage(k0 + 2 + n, c0 + (2 + n) * P, n);
    if (k0 > 0) {  // the interface below the segment
        const TvdFace<V> tf = w_tvd(a.scheme, Wm, dtf, itf, hx_c<V>(H.hlo), hkf);
#pragma unroll
        for (int q = 0; q < NT; q++) {
            V el;
            w_face(tf, Wm, k0 > 1 ? hx_c<V>(H.lo1[q] - H.lo2[q]) : V(0), dkm1[q], dk[q], el, erm[q]);
        }
    }
    int s2 = 0;          // slot of level k + 2
    long long ck = c0;  // offset of level k
    for (int k = k0; k < k1; k++, ck += P, s2 = s2 + 1 == W_RING ? 0 : s2 + 1) {
        // level k + 2: its group is the oldest of the W_STAGE in flight
        __pipeline_wait_prior(W_STAGE - 1);
        const int sf = !SEG || k + 2 < k1 ? s2 : W_RING + (k + 2 - k1);
        const bool in2 = SEG || k + 2 < nz;
        S fk2[NT];
        const double hk2 = in2 ? ring.h(sf) : 0.0;
#pragma unroll
        for (int q = 0; q < NT; q++) fk2[q] = in2 ? ring.f(sf, q) : S(0);
        const V W = Wn;
        const V wk = wkn;
        Wn = (k + 1 < k1 && k + 1 < nz - 1) ? ring.W(s2) : V(0);
        wkn = k + 1 < k1 ? ring.w(s2) : V(0);
        // into the slot of level k + 1, read at k - 1
        stage(k + 2 + W_STAGE, ck + (2 + W_STAGE) * P, s2 == 0 ? W_RING - 1 : s2 - 1);
        const bool inner = k < nz - 1;  // no flux through the surface
        if constexpr (std::is_same<V, double>::value) {
            TvdFace<double> tf{};
            if (inner) tf = w_tvd(a.scheme, W, dtf, itf, hk, hk1);
            const double hn = __fma_rn(-dtkf, __dadd_rn(wk, -wkm1), hk);
            hd[ck] = hn;
            const double coef = __dmul_rn(dtkf, getm_rcp(hn));
            // (w_k - W_k) - (w_{k-1} - W_{k-1}): zero inside a column moved by w itself
            const bool slip = !own_w || k == 0 || !inner;
            const double sl = slip ? __dadd_rn(__dadd_rn(wk, -W), -__dadd_rn(wkm1, -Wm)) : 0.0;
#pragma unroll
            for (int q = 0; q < NT; q++) {
                const double dn = (k + 2 < nz) ? __dadd_rn(fk2[q], -fk1[q]) : 0.0;
                double el = 0.0, er = 0.0;
                if (inner) w_face(tf, W, dkm1[q], dk[q], dn, el, er);
                double num = __dadd_rn(erm[q], -el);
                if (slip) num = __fma_rn(sl, fk[q], num);
                fdst[q][ck] = __fma_rn(coef, num, fk[q]);
                erm[q] = er;
                dkm1[q] = dk[q]; dk[q] = dn;
                fk[q] = fk1[q]; fk1[q] = fk2[q];
            }
        } else {
            // (formed at the surface too, and not used there: no branch)
            const TvdFace<float> tf = w_tvd(a.scheme, W, dtf, itf, hkf, hk1f);
            // (products and sums rounded as written, so that all shapes of the
            // kernel give the same bits)
            const float dh = __fmul_rn(dtkf, wk - wkm1);
            const float den = __fadd_rn(hkf, -dh), sl = (wk - W) - (wkm1 - Wm);
            const double hn = hk - getm_f2d(dh);
            hd[ck] = hn;
#pragma unroll
            for (int q = 0; q < NT; q++) {
                // differences of neighbouring values in the storage type, then
                // narrowed (exact for float storage)
                const float dn = (k + 2 < nz) ? inc_f<S>(fk2[q] - fk1[q]) : 0.f;
                float el = 0.f, er = 0.f;
                if (inner) w_face(tf, W, dkm1[q], dk[q], dn, el, er);
                const float num = __fadd_rn(__fmaf_rn(sl, inc_f<S>(fk[q]), -el), erm[q]);
                fdst[q][ck] = inc_add<S>(fk[q], __fmul_rn(dtkf, num) / den);
                erm[q] = er;
                dkm1[q] = dk[q]; dk[q] = dn;
                fk[q] = fk1[q]; fk1[q] = fk2[q];
            }
        }
        Wm = W; wkm1 = wk;
        hk = hk1; hk1 = hk2;
        hkf = hk1f; hk1f = hx_c<V>(hk2);
    }
    __pipeline_wait_prior(0);  // the ring is free for the next sweep
}

// Largest Courant number over the interfaces above levels k0 .. k1-1 of a
// column where it matters (template :274, :294, :300): -1 when there are none
// or all are clearly below one, which is all the caller asks.  That first
// sweep compares |w_var| dt with 0.999 of the thickness in float, without a
// division; only segments that fail it (or hold a NaN) divide.  A NaN at the
// column's first interface is the result, any other is passed over.
template <typename T, typename V>
__device__ V w_maxcfl(const WPassArgs<T, V>& a, long long c, int k0, int k1, const V* wv, const double* hs)
{
    const long long P = a.plane;
    const int ke = k1 < a.nz ? k1 + 1 : a.nz;  // levels k0 .. ke-1 bound the interfaces
    const float dtf = (float)a.dt;
    float hk = getm_d2f_approx(hs[c + k0 * P]);
    bool low = true;
#pragma unroll 4
    for (int k = k0 + 1; k < ke; k++) {
        const float hk1 = getm_d2f_approx(hs[c + k * P]);
        low = low && fabsf(inc_f<V>(wv[c + k * P])) * dtf < 0.999f * fminf(hk, hk1);
        hk = hk1;
    }
    if (low) return V(-1);
    V cmax = V(-1);
    double hd = hs[c + k0 * P];
    for (int k = k0 + 1; k < ke; k++) {
        const double hd1 = hs[c + k * P];
        V cfl;
        if constexpr (getm_increment_form<V>)
            cfl = fabsf(wv[c + k * P]) * dtf / fminf(getm_d2f_approx(hd), getm_d2f_approx(hd1));
        else
            cfl = fabs(wv[c + k * P]) * a.dt / fmin(hd, hd1);
        if (k == 1 || cfl > cmax) cmax = cfl;
        hd = hd1;
    }
    return cmax;
}

__device__ __forceinline__ int w_iters_from(double cfl)
{
    if (!(cfl > 1.0)) return 1;               // includes nz == 1 and NaN
    double c = ceil(cfl);
    return c > 1e9 ? 1000000000 : (int)c;
}

// One group of NT fields through all sub-steps of the block's columns.  it,
// iters and the rest of a column's state are the same in all its segments;
// every thread of the block comes here and meets the barriers.
template <int NT, bool SEG, typename T, typename V>
__device__ void w_group(const WPassArgs<T, V>& a, long long c, bool touched, int k0, int k1, int t, bool last,
                        const WRing<SEG, T, V>& ring, double* cm)
{
    const int itersmax = 200;
    const V* wv = a.wvar[t];
    int iters = 1, it = 1;
    bool active = touched;
    for (;;) {
        const double* hs = it == 1 ? a.h_in : a.haux;
        const bool ask = active && iters < itersmax;
        double cmax = -1.0;
        if (ask) cmax = (double)w_maxcfl(a, c, k0, k1, wv, hs);
        if constexpr (SEG) {
            cm[threadIdx.y * 32 + threadIdx.x] = cmax;
            __syncthreads();
            cmax = cm[threadIdx.x];
            for (int s = 1; s < (int)blockDim.y; s++) {
                const double m = cm[s * 32 + threadIdx.x];
                if (m > cmax) cmax = m;
            }
        }
        bool go = active;
        if (ask) {
            const int iters_new = w_iters_from(cmax);
            if (iters_new > iters) {
                if (iters_new > itersmax) {
                    iters = itersmax;
                    if (k0 == 0) atomicOr(a.status, 1 << GETM_ERR_ITERS);
                } else {
                    iters = iters_new;
                }
                if (it > 1) {  // start the column again
                    it = 1;
                    go = false;
                }
            }
        }
        // The last sub-step writes the tracer in place and the thickness
        // into haux (the stage's h_in must survive for the next tracer);
        // the last tracer's last sub-step writes the thickness straight
        // into h_out, the pass's result.  The second field's intermediate
        // sub-steps use the upper half of the column work array.
        const T* fs[NT];
        T* fd[NT];
#pragma unroll
        for (int q = 0; q < NT; q++) {
            T* aux = a.faux + q * (a.plane * a.nz);
            fs[q] = it == 1 ? a.f[t + q] : aux;
            fd[q] = it == iters ? a.f[t + q] : aux;
        }
        hs = it == 1 ? a.h_in : a.haux;
        double* hd = it == iters && last ? a.h_out : a.haux;
        WHalo<NT, T> H;
        if constexpr (SEG) {
            if (go) H = w_halo<NT, T, V>(c, a.plane, a.nz, k0, k1, hs, fs, ring);
            __syncthreads();  // every segment has read its neighbours' levels
        }
        if (go) {
            // (not kept across the sweep: registers)
            double itersm1 = 1.0, dtk = a.dt;
            if (iters > 1) {
                itersm1 = 1.0 / iters;
                dtk = a.dt * itersm1;
            }
            w_substep<NT, SEG, T, V>(a, c, k0, k1, wv, hs, fs, hd, fd, dtk, itersm1, H, ring);
            it++;
            active = it <= iters;
        }
        if constexpr (SEG) {
            if (!__syncthreads_or(active)) return;  // (and the writes are done)
        } else {
            if (!active) return;
        }
    }
}

// T: fields; V: velocities.  SEG: a block is 32 columns of one row and
// blockDim.y segments of their levels; else 32 columns of blockDim.y rows.
template <bool SEG, typename T, typename V>
__global__ void __launch_bounds__(SEG ? 32 * W_MAXSEG : 128, SEG ? 2 : (getm_increment_form<V> ? 7 : 4))
    wpass_kernel(WPassArgs<T, V> a)
{
    const int i = blockIdx.x * 32 + threadIdx.x;
    const int j = SEG ? blockIdx.y : blockIdx.y * blockDim.y + threadIdx.y;
    const int k0 = SEG ? threadIdx.y * a.nz / blockDim.y : 0;
    const int k1 = SEG ? (threadIdx.y + 1) * a.nz / blockDim.y : a.nz;
    const bool in = i < a.nx_ && j < a.ny_;
    const long long c = (long long)j * a.nx_ + i;
    const bool touched =
        in && i >= a.ilo && i <= a.ihi && j >= a.jlo && j <= a.jhi && a.tmask[c] == 1 && a.ntracer > 0;
    // a column the pass does not update keeps its thickness (h_out must be a
    // complete field: it is a ping-pong buffer)
    if (in && !touched && a.h_out != a.h_in)
        for (int k = k0; k < k1; k++) a.h_out[c + k * a.plane] = a.h_in[c + k * a.plane];
    if constexpr (SEG) {
        if (!__syncthreads_or(touched)) return;
    } else {
        if (!touched) return;
    }
    // the rings, then (SEG) the segments' largest Courant numbers
    using Ring = WRing<SEG, T, V>;
    const Ring ring(threadIdx.y, threadIdx.x);
    double* cm = reinterpret_cast<double*>(w_smem + blockDim.y * Ring::BYTES);
    // two consecutive fields with the same w_var are stepped together (the
    // sub-step count depends only on w_var and h)
    for (int t = 0; t < a.ntracer;) {
        if (t + 1 < a.ntracer && a.wvar[t + 1] == a.wvar[t]) {
            w_group<2, SEG, T, V>(a, c, touched, k0, k1, t, t + 2 == a.ntracer, ring, cm);
            t += 2;
        } else {
            w_group<1, SEG, T, V>(a, c, touched, k0, k1, t, t + 1 == a.ntracer, ring, cm);
            t++;
        }
    }
}

// Segments per column, of at least four levels each: one where the columns
// alone give 20 warps per SM (FP64 form: 10, the FP64 pipe being busy with
// fewer), more on smaller domains, whose time is the latency of a column's
// sweep.  us with 1 / 2 / 4 segments: 96 x 96 x 20 mixed, two FP64-stored fields,
// 58 / 29 / 18; 244 x 204 x 20 mixed, eight, 221 / 174 / 164; 404 x 304 x 40 mixed,
// two, 133 / 175 / 180 (float fields 80 / 117 / 124); 124 x 104 x 30 FP64, one,
// 83 / 52 / 41; 177 x 135 x 23 FP64, six, 267 / 199 / 272.
static int w_segments(int nx_, int ny_, int nz, bool f64)
{
    const long long strips = (long long)getm_div_up(nx_, 32) * ny_;
    int seg = 1;
    while (seg < W_MAXSEG && strips * seg < (f64 ? 10 : 20) * GETM_SMS && nz / (2 * seg) >= 4) seg *= 2;
    return seg;
}

template <bool SEG, typename T, typename V>
static int launch_wpass(const WPassArgs<T, V>& a, dim3 grid, dim3 block, cudaStream_t stream)
{
    // the staging rings (w_substep); the largest carve-out of shared memory,
    // so that they do not limit the resident warps
    constexpr size_t per = WRing<SEG, T, V>::BYTES + (SEG ? 32 * sizeof(double) : 0);  // per warp
    static std::atomic<unsigned long long> done{0};
    if (!getm_once_per_device(done, [] {
            return cudaFuncSetAttribute(wpass_kernel<SEG, T, V>, cudaFuncAttributePreferredSharedMemoryCarveout, 100) ==
                       cudaSuccess &&
                   cudaFuncSetAttribute(wpass_kernel<SEG, T, V>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)(W_MAXSEG * per)) == cudaSuccess;
        }))
        return GETM_ERR_CUDA;
    wpass_kernel<SEG, T, V><<<grid, block, block.y * per, stream>>>(a);
    GETM_CHECK_LAUNCH();
    return GETM_OK;
}

template <typename T, typename V = T>
static int run_wstage(getm_advection* adv, const getm_grid* tg, const V* w, const V* const* wvar, double dt,
                      const double* h_in, double* h_out, int ntracer, T* const* f, cudaStream_t stream)
{
    WPassArgs<T, V> a;
    memset(&a, 0, sizeof(a));
    a.nx_ = tg->nx_; a.ny_ = tg->ny_; a.nz = tg->kmax - tg->kmin + 1;
    a.plane = (long long)tg->nx_ * tg->ny_;
    a.ilo = tg->halox; a.ihi = tg->halox + (tg->imax - tg->imin);
    a.jlo = tg->haloy; a.jhi = tg->haloy + (tg->jmax - tg->jmin);
    a.tmask = tg->mask; a.w = w; a.dt = dt; a.scheme = adv->scheme; a.status = adv->status;
    a.haux = adv->colbuf[0]; a.faux = (T*)adv->colbuf[1];
    if (a.nz < 1) return GETM_ERR_ARG;
    const int seg = w_segments(a.nx_, a.ny_, a.nz, !getm_increment_form<V>);
    const int rows = seg > 1 ? 1 : getm_tune(GETM_TUNE_COLUMN_ROWS);
    const dim3 block(32, seg > 1 ? seg : rows);
    const dim3 grid(getm_div_up(a.nx_, 32), getm_div_up(a.ny_, rows));
    // Chunks: every chunk starts from h_in; the final h is the last chunk's.
    int done = 0;
    do {
        int n = ntracer - done;
        if (n > GETM_MAX_BATCH) n = GETM_MAX_BATCH;
        a.ntracer = n;
        a.h_in = h_in; a.h_out = h_out;
        for (int t = 0; t < n; t++) { a.wvar[t] = wvar[done + t]; a.f[t] = f[done + t]; }
        const int rc = seg > 1 ? launch_wpass<true, T, V>(a, grid, block, stream)
                               : launch_wpass<false, T, V>(a, grid, block, stream);
        if (rc) return rc;
        done += n;
    } while (done < ntracer);
    return GETM_OK;
}

// Fused Strang split for any form (see getm_advection_apply_3d_batch): T
// the fields, V the velocities.
template <typename T, typename V = T>
static int apply_3d_batch_impl(getm_advection* adv, getm_grid* tgrid, getm_grid* ugrid, getm_grid* vgrid,
                               int ufirst, const V* u, const V* v, const V* w, const V* const* w_var,
                               const double* Ah_u, const double* Ah_v, double timestep, double* h,
                               const double* hu, const double* hv, int ntracer, T* const* vars,
                               cudaStream_t stream)
{
    if (!adv) return GETM_OK;
    if (!tgrid || !w || !h || ntracer < 1 || !vars) return GETM_ERR_ARG;
    const int nz = tgrid->kmax - tgrid->kmin + 1;
    HPassArgs<T, V> ax, ay;
    int rc = hpass_setup<T, V>(ax, 1, adv, tgrid, ugrid, nz, u, Ah_u, 0.5 * timestep, hu);
    if (rc) return rc;
    if ((rc = hpass_setup<T, V>(ay, 2, adv, tgrid, vgrid, nz, v, Ah_v, 0.5 * timestep, hv))) return rc;
    const size_t n3 = (size_t)ax.plane * nz;
    if ((rc = adv_reserve(adv, n3, ntracer))) return rc;

    const V* wv[GETM_MAX_BATCH * 8];
    const T* fin[GETM_MAX_BATCH * 8];
    T* fout[GETM_MAX_BATCH * 8];
    T* tmp[GETM_MAX_BATCH * 8];
    for (int t = 0; t < ntracer; t++) {
        wv[t] = (w_var && w_var[t]) ? w_var[t] : w;
        tmp[t] = (T*)adv->tmp[t];
    }

    HPassArgs<T, V>* first = ufirst ? &ax : &ay;
    const int dfirst = ufirst ? 1 : 2;
    HPassArgs<T, V>* second = ufirst ? &ay : &ax;
    const int dsecond = ufirst ? 2 : 1;
    double* A = adv->hbuf[0];
    double* B = adv->hbuf[1];

    // adv1(dt/2): vars -> tmp, h -> A   (operators.py:165-170)
    for (int t = 0; t < ntracer; t++) { fin[t] = vars[t]; fout[t] = tmp[t]; }
    if ((rc = run_hstage<T, V>(*first, dfirst, h, A, ntracer, fin, fout, stream))) return rc;
    // adv2(dt/2): tmp -> vars, A -> B   (:171-175)
    for (int t = 0; t < ntracer; t++) { fin[t] = tmp[t]; fout[t] = vars[t]; }
    if ((rc = run_hstage<T, V>(*second, dsecond, A, B, ntracer, fin, fout, stream))) return rc;
    // w(dt): vars in place, B -> A      (:176-182)
    if ((rc = run_wstage<T, V>(adv, tgrid, w, wv, timestep, B, A, ntracer, vars, stream))) return rc;
    // adv2(dt/2): vars -> tmp, A -> B   (:183-188)
    for (int t = 0; t < ntracer; t++) { fin[t] = vars[t]; fout[t] = tmp[t]; }
    if ((rc = run_hstage<T, V>(*second, dsecond, A, B, ntracer, fin, fout, stream))) return rc;
    // adv1(dt/2): tmp -> vars, B -> h   (:189-193)
    for (int t = 0; t < ntracer; t++) { fin[t] = tmp[t]; fout[t] = vars[t]; }
    if ((rc = run_hstage<T, V>(*first, dfirst, B, h, ntracer, fin, fout, stream))) return rc;
    return GETM_OK;
}

// ---------------------------------------------------------------------------
// C ABI
// ---------------------------------------------------------------------------
extern "C" int getm_advection_uv_calculate(int direction, int nk, getm_advection* adv,
                                           getm_grid* tgrid, getm_grid* ugrid, const double* u,
                                           const double* Ah, double timestep, double* h,
                                           const double* hu, double* var, cudaStream_t stream)
{
    if (!adv) return GETM_OK;  // wrapper.F90:227 returns silently without a scheme
    if ((direction != 1 && direction != 2) || nk < 1 || !h || !var) return GETM_ERR_ARG;
    HPassArgs<double> a;
    int rc = hpass_setup(a, direction, adv, tgrid, ugrid, nk, u, Ah, timestep, hu);
    if (rc) return rc;
    const size_t n3 = (size_t)a.plane * nk;
    if ((rc = adv_reserve(adv, n3, 1))) return rc;
    const double* fin[1] = {var};
    double* fout[1] = {adv->tmp[0]};
    if ((rc = run_hstage(a, direction, h, adv->hbuf[0], 1, fin, fout, stream))) return rc;
    // in-place semantics of the reference: copy the results back
    if (cudaMemcpyAsync(var, adv->tmp[0], n3 * sizeof(double), cudaMemcpyDeviceToDevice, stream) != cudaSuccess) return GETM_ERR_CUDA;
    if (cudaMemcpyAsync(h, adv->hbuf[0], n3 * sizeof(double), cudaMemcpyDeviceToDevice, stream) != cudaSuccess) return GETM_ERR_CUDA;
    return GETM_OK;
}

extern "C" int getm_advection_w_calculate(getm_advection* adv, getm_grid* tgrid, const double* w,
                                          const double* w_var, double timestep, double* h,
                                          double* var, cudaStream_t stream)
{
    if (!adv) return GETM_OK;  // wrapper.F90:265
    if (!tgrid || !w || !w_var || !h || !var || !tgrid->mask) return GETM_ERR_ARG;
    const int nz = tgrid->kmax - tgrid->kmin + 1;
    const size_t n3 = (size_t)tgrid->nx_ * tgrid->ny_ * nz;
    int rc = adv_reserve(adv, n3, 0);
    if (rc) return rc;
    const double* wv[1] = {w_var};
    double* f[1] = {var};
    if ((rc = run_wstage<double>(adv, tgrid, w, wv, timestep, h, adv->hbuf[0], 1, f, stream))) return rc;
    if (cudaMemcpyAsync(h, adv->hbuf[0], n3 * sizeof(double), cudaMemcpyDeviceToDevice, stream) != cudaSuccess) return GETM_ERR_CUDA;
    return GETM_OK;
}

extern "C" int getm_advection_apply_3d_batch(getm_advection* adv, getm_grid* tgrid,
                                             getm_grid* ugrid, getm_grid* vgrid, int ufirst,
                                             const double* u, const double* v, const double* w,
                                             const double* const* w_var, const double* Ah_u,
                                             const double* Ah_v, double timestep, double* h,
                                             const double* hu, const double* hv, int ntracer,
                                             double* const* vars, cudaStream_t stream)
{
    return apply_3d_batch_impl<double>(adv, tgrid, ugrid, vgrid, ufirst, u, v, w, w_var, Ah_u, Ah_v, timestep, h,
                                       hu, hv, ntracer, vars, stream);
}

extern "C" int getm_advection_apply_3d_batch_f32(getm_advection* adv, getm_grid* tgrid,
                                                 getm_grid* ugrid, getm_grid* vgrid, int ufirst,
                                                 const float* u, const float* v, const float* w,
                                                 const float* const* w_var, const double* Ah_u,
                                                 const double* Ah_v, double timestep, double* h,
                                                 const double* hu, const double* hv, int ntracer,
                                                 float* const* vars, cudaStream_t stream)
{
    return apply_3d_batch_impl<float>(adv, tgrid, ugrid, vgrid, ufirst, u, v, w, w_var, Ah_u, Ah_v, timestep, h,
                                      hu, hv, ntracer, vars, stream);
}

extern "C" int getm_advection_apply_3d_batch_f64s(getm_advection* adv, getm_grid* tgrid,
                                                  getm_grid* ugrid, getm_grid* vgrid, int ufirst,
                                                  const float* u, const float* v, const float* w,
                                                  const float* const* w_var, const double* Ah_u,
                                                  const double* Ah_v, double timestep, double* h,
                                                  const double* hu, const double* hv, int ntracer,
                                                  double* const* vars, cudaStream_t stream)
{
    return apply_3d_batch_impl<double, float>(adv, tgrid, ugrid, vgrid, ufirst, u, v, w, w_var, Ah_u, Ah_v,
                                              timestep, h, hu, hv, ntracer, vars, stream);
}

template <typename T, typename V = T>
static int uv_pass_impl(int direction, int nk, getm_advection* adv, getm_grid* tgrid, getm_grid* ugrid,
                        const V* u, const double* Ah, double timestep, const double* h_in, double* h_out,
                        const double* hu, int ntracer, const T* const* fin, T* const* fout, cudaStream_t stream)
{
    if (!adv || (direction != 1 && direction != 2) || nk < 1 || !h_in || !h_out || ntracer < 0) return GETM_ERR_ARG;
    if (ntracer > 0 && (!fin || !fout)) return GETM_ERR_ARG;
    if (h_in == h_out) return GETM_ERR_ARG;
    for (int t = 0; t < ntracer; t++)
        if (!fin[t] || !fout[t] || (const void*)fin[t] == (const void*)fout[t]) return GETM_ERR_ARG;
    HPassArgs<T, V> a;
    int rc = hpass_setup<T, V>(a, direction, adv, tgrid, ugrid, nk, u, Ah, timestep, hu);
    if (rc) return rc;
    return run_hstage<T, V>(a, direction, h_in, h_out, ntracer, fin, fout, stream);
}

extern "C" int getm_advection_uv_pass(int direction, int nk, getm_advection* adv, getm_grid* tgrid,
                                      getm_grid* ugrid, const double* u, const double* Ah, double timestep,
                                      const double* h_in, double* h_out, const double* hu, int ntracer,
                                      const double* const* var_in, double* const* var_out, cudaStream_t stream)
{
    return uv_pass_impl<double>(direction, nk, adv, tgrid, ugrid, u, Ah, timestep, h_in, h_out, hu, ntracer, var_in,
                                var_out, stream);
}

extern "C" int getm_advection_uv_pass_f32(int direction, int nk, getm_advection* adv, getm_grid* tgrid,
                                          getm_grid* ugrid, const float* u, const double* Ah, double timestep,
                                          const double* h_in, double* h_out, const double* hu, int ntracer,
                                          const float* const* var_in, float* const* var_out, cudaStream_t stream)
{
    return uv_pass_impl<float>(direction, nk, adv, tgrid, ugrid, u, Ah, timestep, h_in, h_out, hu, ntracer, var_in,
                               var_out, stream);
}

extern "C" int getm_advection_uv_pass_f64s(int direction, int nk, getm_advection* adv, getm_grid* tgrid,
                                           getm_grid* ugrid, const float* u, const double* Ah, double timestep,
                                           const double* h_in, double* h_out, const double* hu, int ntracer,
                                           const double* const* var_in, double* const* var_out,
                                           cudaStream_t stream)
{
    return uv_pass_impl<double, float>(direction, nk, adv, tgrid, ugrid, u, Ah, timestep, h_in, h_out, hu, ntracer,
                                       var_in, var_out, stream);
}

// D0: the column heights before the first pass (D itself, or the caller's
// field); D: those after the last.
static int advection_2d_impl(getm_advection* adv, getm_grid* tgrid, getm_grid* ugrid, getm_grid* vgrid,
                             int ufirst, int split, const double* u, const double* v, const double* Ah_u,
                             const double* Ah_v, double timestep, const double* D0, double* D, const double* DU,
                             const double* DV, double* var, int increment, cudaStream_t stream)
{
    if (!adv) return GETM_OK;
    if (!D0 || !D || !var || split < 1 || split > 3) return GETM_ERR_ARG;
    HPassArgs<double> ax, ay;
    int rc = hpass_setup(ax, 1, adv, tgrid, ugrid, 1, u, Ah_u, timestep, DU, increment);
    if (rc) return rc;
    if ((rc = hpass_setup(ay, 2, adv, tgrid, vgrid, 1, v, Ah_v, timestep, DV, increment))) return rc;
    const size_t n2 = (size_t)ax.plane;
    if ((rc = adv_reserve(adv, n2, 1))) return rc;
    HPassArgs<double>* p1 = ufirst ? &ax : &ay;
    HPassArgs<double>* p2 = ufirst ? &ay : &ax;
    const int d1 = ufirst ? 1 : 2, d2 = ufirst ? 2 : 1;
    // (the vertical pass's work array, idle here, is the second buffer: a handle
    // that a call with one field has sized allocates nothing more)
    double* const T[2] = {adv->tmp[0], adv->colbuf[1]};
    double* A = adv->hbuf[0];
    double* B = adv->hbuf[1];
    const double* fin[1];
    double* fout[1];
    // Sequence of (pass, dt factor): var->T0->T1->...->var and D0->A->B->...->D
    int seq_n = 0;
    int seq_dir[4];
    double seq_dt[4];
    HPassArgs<double>* seq_a[4];
    if (split == 1) {          // FULL: adv1(dt), adv2(dt)
        seq_a[0] = p1; seq_dir[0] = d1; seq_dt[0] = timestep;
        seq_a[1] = p2; seq_dir[1] = d2; seq_dt[1] = timestep;
        seq_n = 2;
    } else if (split == 2) {   // HALF: adv1(dt/2), adv2(dt), adv1(dt/2)
        seq_a[0] = p1; seq_dir[0] = d1; seq_dt[0] = 0.5 * timestep;
        seq_a[1] = p2; seq_dir[1] = d2; seq_dt[1] = timestep;
        seq_a[2] = p1; seq_dir[2] = d1; seq_dt[2] = 0.5 * timestep;
        seq_n = 3;
    } else {                   // HALF_ALWAYS: adv1/2, adv2/2, adv2/2, adv1/2
        seq_a[0] = p1; seq_dir[0] = d1; seq_dt[0] = 0.5 * timestep;
        seq_a[1] = p2; seq_dir[1] = d2; seq_dt[1] = 0.5 * timestep;
        seq_a[2] = p2; seq_dir[2] = d2; seq_dt[2] = 0.5 * timestep;
        seq_a[3] = p1; seq_dir[3] = d1; seq_dt[3] = 0.5 * timestep;
        seq_n = 4;
    }
    const double* hsrc = D0;
    const double* fsrc = var;
    for (int s = 0; s < seq_n; s++) {
        double* hdst = (s == seq_n - 1) ? D : ((s % 2 == 0) ? A : B);
        double* fdst = (s == seq_n - 1) ? var : T[s % 2];
        seq_a[s]->dt = seq_dt[s];
        seq_a[s]->dtf = (float)seq_dt[s];
        fin[0] = fsrc; fout[0] = fdst;
        if ((rc = run_hstage(*seq_a[s], seq_dir[s], hsrc, hdst, 1, fin, fout, stream))) return rc;
        hsrc = hdst;
        fsrc = fdst;
    }
    return GETM_OK;
}

int getm_advection_2d_passes(getm_advection* adv, getm_grid* tgrid, getm_grid* ugrid, getm_grid* vgrid,
                             int ufirst, const double* u, const double* v, double timestep, double* D,
                             const double* DU, const double* DV, double* var, int increment,
                             Advection2DPasses* out)
{
    if (!adv || !D || !var || !out) return GETM_ERR_ARG;
    HPassArgs<double> ax, ay;
    int rc = hpass_setup(ax, 1, adv, tgrid, ugrid, 1, u, nullptr, timestep, DU, increment);
    if (rc) return rc;
    if ((rc = hpass_setup(ay, 2, adv, tgrid, vgrid, 1, v, nullptr, timestep, DV, increment))) return rc;
    if ((rc = adv_reserve(adv, (size_t)ax.plane, 1))) return rc;
    out->pass[0] = ufirst ? ax : ay;
    out->pass[1] = ufirst ? ay : ax;
    out->dir[0] = ufirst ? 1 : 2;
    out->dir[1] = ufirst ? 2 : 1;
    HPassArgs<double>& p1 = out->pass[0];
    HPassArgs<double>& p2 = out->pass[1];
    p1.ntracer = p2.ntracer = 1;
    p1.h_in = D; p1.h_out = adv->hbuf[0]; p1.fin[0] = var; p1.fout[0] = adv->tmp[0];
    p2.h_in = adv->hbuf[0]; p2.h_out = D; p2.fin[0] = adv->tmp[0]; p2.fout[0] = var;
    return GETM_OK;
}

extern "C" int getm_advection_2d(getm_advection* adv, getm_grid* tgrid, getm_grid* ugrid,
                                 getm_grid* vgrid, int ufirst, int split, const double* u,
                                 const double* v, const double* Ah_u, const double* Ah_v,
                                 double timestep, double* D, const double* DU, const double* DV,
                                 double* var, cudaStream_t stream)
{
    return advection_2d_impl(adv, tgrid, ugrid, vgrid, ufirst, split, u, v, Ah_u, Ah_v, timestep, D, D, DU, DV, var,
                             0, stream);
}

extern "C" int getm_advection_2d_mixed(getm_advection* adv, getm_grid* tgrid, getm_grid* ugrid,
                                       getm_grid* vgrid, int ufirst, int split, const double* u,
                                       const double* v, const double* Ah_u, const double* Ah_v,
                                       double timestep, double* D, const double* DU, const double* DV,
                                       double* var, cudaStream_t stream)
{
    return advection_2d_impl(adv, tgrid, ugrid, vgrid, ufirst, split, u, v, Ah_u, Ah_v, timestep, D, D, DU, DV, var,
                             1, stream);
}

extern "C" int getm_advection_2d_from(getm_advection* adv, getm_grid* tgrid, getm_grid* ugrid, getm_grid* vgrid,
                                      int ufirst, int split, const double* u, const double* v, const double* Ah_u,
                                      const double* Ah_v, double timestep, const double* D0, double* D,
                                      const double* DU, const double* DV, double* var, int mixed,
                                      cudaStream_t stream)
{
    return advection_2d_impl(adv, tgrid, ugrid, vgrid, ufirst, split, u, v, Ah_u, Ah_v, timestep, D0, D, DU, DV, var,
                             mixed != 0, stream);
}

// ---------------------------------------------------------------------------
// Allocation-free variant of the 2D advection split
// ---------------------------------------------------------------------------
// getm_advection_2d keeps its ping-pong buffers in a handle that allocates
// them with cudaMalloc on first use.  Some callers cannot allow that: a host
// model that hands all device memory to its own pool allocator at start-up
// (a library cudaMalloc then fails or breaks the pool's accounting), and
// drivers that must not let a library call synchronize the device (cudaMalloc
// and cudaFree may do so implicitly).  getm_advection_2d_noalloc takes the
// scheme instead of a handle and keeps its three work buffers (tracer
// ping-pong copy and two column-height buffers) in one file-scope device
// array of fixed size, so it allocates nothing.
//
// Limits and sharing rules:
// * the domain may have at most GETM_NOALLOC_MAX_POINTS points including
//   halos (nx_ * ny_); larger domains get GETM_ERR_TOO_LARGE and nothing runs;
// * every GPU that loads the library holds the 3 * 2^20 doubles (24 MiB)
//   until the process exits;
// * all calls share the one array, which keeps the previous call's contents.
//   Nothing in it has to start at zero: every pass writes all points of the
//   buffer it produces before the next pass reads them.  Calls that overlap on
//   the GPU (different streams, or different host threads without ordering)
//   race on the array and corrupt each other's results;
// * the first call on a device looks up the array's device address with
//   cudaGetSymbolAddress (once per device, with that device current).  Make
//   that first call before any stream capture.
#include <mutex>

#define GETM_NOALLOC_MAX_POINTS (1 << 20)
#define GETM_NOALLOC_MAX_DEVICES 64

static __device__ __align__(256) double g_noalloc_scratch[3 * GETM_NOALLOC_MAX_POINTS];
static double* g_noalloc_ptr[GETM_NOALLOC_MAX_DEVICES];
static std::mutex g_noalloc_mutex;

// Device address of the scratch array for the current device.
static int noalloc_scratch(double** out)
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return GETM_ERR_CUDA;
    if (dev < 0 || dev >= GETM_NOALLOC_MAX_DEVICES) return GETM_ERR_ARG;
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (!g_noalloc_ptr[dev]) {
        void* p = NULL;
        cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess || p == NULL) return GETM_ERR_CUDA;
        g_noalloc_ptr[dev] = (double*)p;
    }
    *out = g_noalloc_ptr[dev];
    return GETM_OK;
}

extern "C" int getm_advection_2d_noalloc(int scheme, getm_grid* tgrid, getm_grid* ugrid, getm_grid* vgrid,
                                         int ufirst, int split, const double* u, const double* v,
                                         const double* Ah_u, const double* Ah_v, double timestep, double* D,
                                         const double* DU, const double* DV, double* var, cudaStream_t stream)
{
    if (scheme < GETM_SCHEME_HSIMT || scheme > GETM_SCHEME_UPSTREAM) return GETM_ERR_ARG;
    if (!tgrid || !D || !var || split < 1 || split > 3) return GETM_ERR_ARG;
    const long long npoints = (long long)tgrid->nx_ * tgrid->ny_;
    if (npoints > GETM_NOALLOC_MAX_POINTS) return GETM_ERR_TOO_LARGE;
    getm_advection adv;  // scheme only: lives on the host stack, owns nothing
    memset(&adv, 0, sizeof(adv));
    adv.scheme = scheme;
    HPassArgs<double> ax, ay;
    int rc = hpass_setup(ax, 1, &adv, tgrid, ugrid, 1, u, Ah_u, timestep, DU);
    if (rc) return rc;
    if ((rc = hpass_setup(ay, 2, &adv, tgrid, vgrid, 1, v, Ah_v, timestep, DV))) return rc;
    double* scratch = NULL;
    if ((rc = noalloc_scratch(&scratch))) return rc;
    double* T = scratch;
    double* A = scratch + GETM_NOALLOC_MAX_POINTS;
    double* B = scratch + 2 * GETM_NOALLOC_MAX_POINTS;
    HPassArgs<double>* p1 = ufirst ? &ax : &ay;
    HPassArgs<double>* p2 = ufirst ? &ay : &ax;
    const int d1 = ufirst ? 1 : 2, d2 = ufirst ? 2 : 1;
    int seq_n = 0;
    int seq_dir[4];
    double seq_dt[4];
    HPassArgs<double>* seq_a[4];
    if (split == 1) {  // FULL (operators.py:76-79)
        seq_a[0] = p1; seq_dir[0] = d1; seq_dt[0] = timestep;
        seq_a[1] = p2; seq_dir[1] = d2; seq_dt[1] = timestep;
        seq_n = 2;
    } else if (split == 2) {  // HALF (operators.py:80-85)
        seq_a[0] = p1; seq_dir[0] = d1; seq_dt[0] = 0.5 * timestep;
        seq_a[1] = p2; seq_dir[1] = d2; seq_dt[1] = timestep;
        seq_a[2] = p1; seq_dir[2] = d1; seq_dt[2] = 0.5 * timestep;
        seq_n = 3;
    } else {  // HALF_ALWAYS (operators.py:86-93)
        seq_a[0] = p1; seq_dir[0] = d1; seq_dt[0] = 0.5 * timestep;
        seq_a[1] = p2; seq_dir[1] = d2; seq_dt[1] = 0.5 * timestep;
        seq_a[2] = p2; seq_dir[2] = d2; seq_dt[2] = 0.5 * timestep;
        seq_a[3] = p1; seq_dir[3] = d1; seq_dt[3] = 0.5 * timestep;
        seq_n = 4;
    }
    const double* fin[1];
    double* fout[1];
    const double* hsrc = D;
    double* fsrc = var;
    for (int s = 0; s < seq_n; s++) {
        double* hdst = (s == seq_n - 1) ? D : ((s % 2 == 0) ? A : B);
        double* fdst = (fsrc == var) ? T : var;
        seq_a[s]->dt = seq_dt[s];
        seq_a[s]->dtf = (float)seq_dt[s];
        fin[0] = fsrc;
        fout[0] = fdst;
        if ((rc = run_hstage(*seq_a[s], seq_dir[s], hsrc, hdst, 1, fin, fout, stream))) return rc;
        hsrc = hdst;
        fsrc = fdst;
    }
    if (fsrc != var) {
        if (cudaMemcpyAsync(var, fsrc, (size_t)npoints * sizeof(double), cudaMemcpyDeviceToDevice, stream) != cudaSuccess)
            return GETM_ERR_CUDA;
    }
    return GETM_OK;
}
