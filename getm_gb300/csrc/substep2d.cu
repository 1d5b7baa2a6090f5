// One split-explicit 2D substep as four kernels for sm_103a.
//
// A 2D substep of pygetm's Simulation.advance that is not followed by a 3D
// (macro) step (python/pygetm/simulation.py:1033-1304: advance_depth_integrated,
// advance_surface_elevation, update_depth, update_depth_integrated_diagnostics,
// the surface pressure gradient and the wind-stress interpolation) is some
// twenty operations on fields of one horizontal plane.  Launched one by one
// they leave GB300 idle between launches: each reads and writes ~10^5 points,
// a microsecond of work behind several microseconds of launch and drain.
//
// The operations depend on one another through neighbouring points only, in
// seven phases:
//   1  transport update of the first direction (U or V, alternating)
//   2  Coriolis term from it, then the second direction's update
//   3  Coriolis term from the second, cumulative transports, zo = z and the
//      surface elevation update
//   4  depths (update_depth, 2D part), fwf = pe, wind stress interpolation
//   5  velocities and advection velocities, copies of the depths advected
//      by the momentum advection, surface pressure gradient
//   6  bottom friction, first pass of the U and V momentum advection
//   7  second pass of both, forming each cell's advection term from its
//      transport change as the pass finishes the cell (reconstruct)
// For one domain, a kernel forms what its tile needs of the phases before it
// at the tile's edge once more (a row and a column), so that phases 1 and 2
// are one launch and 3 to 5 another; the two advection passes are one launch
// each (substep_* kernels below).  For many domains at once, one cooperative
// launch walks through the seven phases with grid-wide barriers between them
// (substep_batch_kernel at the end).  Every operation is the same device
// function the separate kernels run (split2d_ops.cuh, advection_passes.cuh),
// so results are bitwise the same.
//
// The batch kernel's barrier is a counter and a generation word in global
// memory.  Its wait is bounded: after about a second it sets the error word,
// every block returns, and later launches return at once until the host clears
// the word.
#include <string.h>

#include <algorithm>
#include <mutex>
#include <type_traits>

#include "advection_passes.cuh"
#include "split2d_ops.cuh"

namespace {

constexpr int SS_BY = 16;
constexpr int SS_THREADS = 32 * SS_BY;
constexpr unsigned SS_SPIN_LIMIT = 1u << 22;

__host__ __device__ inline int div_up(int a, int b) { return (a + b - 1) / b; }

struct SubstepArgs {
    int nx, ny, halox, haloy;
    int ufirst, accumulate, friction;
    int early;                   // the next kernel is launched as each block begins
    double dt, idt;
    double* time;
    Transport2DArgs tr[2];       // [0]: U, [1]: V
    double* cor_out[2];          // Coriolis terms corU, corV (read by tr[].cor)
    const double* corf[2];       // Coriolis parameter on U, V
    double *Ucum, *Vcum;
    const int* mT;
    const double *dyU, *dxV, *iareaT;
    double *z, *zo, *fwf;
    const double* pe;
    DepthArgs depth;
    VelArgs vel;
    FricArgs fric;
    SpgArgs spg;
    const double *taux, *tauy;
    double *tausx, *tausy;
    Advection2DPasses adv[2];    // momentum advection of U and V
    const double* Dsrc[2];       // U.D, V.D
    double* advD[2];             // the advections' thickness arrays
    double* advvar[2];           // advU, advV
    const double* Uo[2];         // U, V
    unsigned* sync;              // [0] barrier arrivals, [1] blocks done, [2] error
};

static_assert(SS_BY == HY_BY, "the y passes run on the kernel's 32 x 16 blocks");

union SubstepSmem {
    double szh[SS_BY + 2][UD_BX + 2];
    YIncSmem<double, float> yf;   // mixed form
    YIncSmem<double, double> yd;  // FP64 form
};

__device__ __forceinline__ unsigned ld_acquire(const unsigned* p)
{
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void red_release_add(unsigned* p, unsigned v)
{
    asm volatile("red.release.gpu.global.add.u32 [%0], %1;" : : "l"(p), "r"(v) : "memory");
}

// Grid-wide barrier k of a launch: thread 0 of every block adds one arrival
// and waits until the count reaches k blocks per block; false when the wait
// gave up or another block reported an error (the caller returns).  The
// count only grows during a launch; the last block to leave the kernel
// resets it (grid_exit) for the next launch on the stream.  Ordering: the
// block barrier orders the block's writes before thread 0's release
// arrival, and thread 0's acquire load followed by the block barrier orders
// the other blocks' writes before every thread's later reads.
__device__ __forceinline__ bool grid_barrier(unsigned* sync, unsigned& target, int& s_ok)
{
    __syncthreads();
    if (threadIdx.x == 0 && threadIdx.y == 0) {
        target += gridDim.x;
        red_release_add(&sync[0], 1u);
        int ok = 1;
        unsigned it = 0;
        while (ld_acquire(&sync[0]) < target) {
            if (++it > SS_SPIN_LIMIT) {
                atomicExch(&sync[2], 1u);
                ok = 0;
                break;
            }
            if ((it & 255u) == 0 && ld_acquire(&sync[2]) != 0) {  // another block gave up
                ok = 0;
                break;
            }
        }
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}

__device__ __forceinline__ void grid_exit(unsigned* sync)
{
    if (threadIdx.x == 0 && threadIdx.y == 0) {
        __threadfence();
        if (atomicAdd(&sync[1], 1u) == gridDim.x - 1) {
            atomicExch(&sync[0], 0u);
            atomicExch(&sync[1], 0u);
        }
    }
}

// reconstruct_transport_change (momentum.F90:323-340) of a cell as soon as
// the last advection pass has finished it: un = (un hn - Uo) / dt on rows
// jlo..jhi (the same expression as reconstruct_point)
struct ReconstructEpi {
    double* un;
    const double* Uo;
    double idt;
    int jlo, jhi;
    __device__ __forceinline__ void operator()(long long p, int j, double fn, double hn) const
    {
        if (j < jlo || j > jhi) return;
        un[p] = (fn * hn - Uo[p]) * idt;
    }
};

// Coriolis term on the other velocity grid from the transport of direction
// d (momentum.py:1127-1148): U -> V with offsets (1, 0), negated; V -> U
// with offsets (0, 1).
template <typename C>
__device__ __forceinline__ void coriolis_from(const SubstepArgs& a, int d, int i, int j, const double* src)
{
    const int o = 1 - d;
    coriolis_2d_point<C>(a.nx, a.ny, d == 0 ? 1 : 0, d == 0 ? 0 : 1, src, a.corf[o], a.cor_out[o], d == 0, i,
                         j);
}

// The pointwise operations of phase ph + 1 (a constant where this is inlined)
// at point p = (i, j); d1: the direction updated first.  Phase 4 has its
// depth tiles besides, phase 6 its advection passes.
template <bool MIXED>
__device__ __forceinline__ void phase_point(const SubstepArgs& a, int ph, int d1, int i, int j, int p,
                                            bool spg = true)
{
    using C = typename std::conditional<MIXED, float, double>::type;
    const int nx = a.nx, ny = a.ny, d2 = 1 - d1;
    const bool interior = i >= a.halox && i < nx - a.halox && j >= a.haloy && j < ny - a.haloy;
    switch (ph) {
    case 0:
        if (interior) transport_2d_point<MIXED>(a.tr[d1], a.dt, p);
        break;
    case 1:
        coriolis_from<C>(a, d1, i, j, a.tr[d1].U);
        if (interior) transport_2d_point<MIXED>(a.tr[d2], a.dt, p);
        break;
    case 2:
        coriolis_from<C>(a, d2, i, j, a.tr[d2].U);
        if (a.accumulate) accumulate_2d_point(a.tr[0].U, a.tr[1].U, a.Ucum, a.Vcum, p);
        surface_elevation_fused_point(nx, ny, a.halox, a.haloy, a.mT, a.dyU, a.dxV, a.iareaT, a.z, a.zo,
                                      a.tr[0].U, a.tr[1].U, a.fwf, a.dt, i, j);
        break;
    case 3:
        a.fwf[p] = a.pe[p];
        if (i < nx - 1) interp_pair_point<double>(a.taux, a.tausx, p, 1, 0);
        if (j < ny - 1) interp_pair_point<double>(a.tauy, a.tausy, p, nx, 0);
        break;
    case 4:
        momentum_2d_velocities_point<C>(a.vel, i, j);
        a.advD[0][p] = a.Dsrc[0][p];
        a.advD[1][p] = a.Dsrc[1][p];
        if (spg && interior) spg_point<MIXED>(a.spg, p);
        break;
    default:
        momentum_2d_friction_point<C>(a.fric, i, j);
        break;
    }
}

static_assert(sizeof(SubstepArgs) <= 4096, "kernel parameter block");

constexpr int SS_MAX_DEVICES = 64;

// The kernels' arguments for one domain from its fields and handles; a
// GETM_* status.
int substep_args(SubstepArgs& a, const getm_split2d_fields* f, int nx, int ny, int halox, int haloy, int mixed,
                 int ufirst, int accumulate, int friction, double timestep, double Dmin, double Dcrit,
                 getm_advection* uadv, getm_grid* ugrid, getm_grid* uugrid, getm_grid* uvgrid, int uadv_ufirst,
                 getm_advection* vadv, getm_grid* vgrid, getm_grid* vugrid, getm_grid* vvgrid, int vadv_ufirst)
{
    if (!f || nx < 2 || ny < 2 || halox < 1 || haloy < 1 || !(timestep > 0.0) || !uadv || !vadv) return GETM_ERR_ARG;
    if ((long long)(nx + 1) * (ny + 1) >= (1ll << 30)) return GETM_ERR_ARG;
    const void* ptrs[] = {f->mask_t, f->H_t, f->iarea_t, f->z, f->zo, f->D_t, f->Dclip_t, f->work_t, f->fwf, f->pe,
                          f->sp, f->taux, f->tauy,
                          f->mask_u, f->H_u, f->dy_u, f->idx_u, f->cor_u, f->z0b_u, f->D_u, f->alpha_u, f->work_u,
                          f->U, f->dpdx, f->tausx, f->corU, f->advU, f->diffU, f->dampU, f->SxA, f->SxB, f->SxD,
                          f->SxF, f->ru, f->u1, f->Ucum, f->advD_u, f->uua, f->uva,
                          f->mask_v, f->H_v, f->dx_v, f->idy_v, f->cor_v, f->z0b_v, f->D_v, f->alpha_v, f->work_v,
                          f->V, f->dpdy, f->tausy, f->corV, f->advV, f->diffV, f->dampV, f->SyA, f->SyB, f->SyD,
                          f->SyF, f->rv, f->v1, f->Vcum, f->advD_v, f->vua, f->vva,
                          f->mask_x, f->H_x, f->D_x, f->work_x, f->D_uu, f->D_uv, f->D_vu, f->D_vv, f->sync};
    for (const void* q : ptrs)
        if (!q) return GETM_ERR_ARG;
    memset(&a, 0, sizeof(a));
    a.nx = nx; a.ny = ny; a.halox = halox; a.haloy = haloy;
    a.ufirst = ufirst != 0; a.accumulate = accumulate != 0; a.friction = friction != 0;
    a.dt = timestep; a.idt = 1.0 / timestep;
    a.time = f->time;
    a.tr[0] = Transport2DArgs{f->mask_u, f->alpha_u, f->D_u, f->dpdx, f->tausx, f->corU, f->advU, f->diffU,
                              f->dampU, f->SxA, f->SxB, f->SxD, f->SxF, f->ru, f->U};
    a.tr[1] = Transport2DArgs{f->mask_v, f->alpha_v, f->D_v, f->dpdy, f->tausy, f->corV, f->advV, f->diffV,
                              f->dampV, f->SyA, f->SyB, f->SyD, f->SyF, f->rv, f->V};
    a.cor_out[0] = f->corU; a.cor_out[1] = f->corV;
    a.corf[0] = f->cor_u; a.corf[1] = f->cor_v;
    a.Ucum = f->Ucum; a.Vcum = f->Vcum;
    a.mT = f->mask_t; a.dyU = f->dy_u; a.dxV = f->dx_v; a.iareaT = f->iarea_t;
    a.z = f->z; a.zo = f->zo; a.fwf = f->fwf; a.pe = f->pe;
    a.depth = DepthArgs{nx, ny, Dmin, Dcrit, 1.0 / (Dcrit - 2 * Dmin), f->z, f->zo, f->H_t, f->H_u, f->H_v, f->H_x,
                        f->mask_t, f->mask_u, f->mask_v, f->mask_x, f->D_t, f->Dclip_t, f->work_t, f->work_u,
                        f->D_u, f->alpha_u, f->work_v, f->D_v, f->alpha_v, f->work_x, f->D_x, f->D_uu, f->D_vv,
                        f->D_uv, f->D_vu};
    a.vel = VelArgs{nx, ny, f->U, f->V, f->D_u, f->D_v, f->D_uu, f->D_uv, f->D_vu, f->D_vv, f->u1, f->v1, f->advU,
                    f->advV, f->uua, f->uva, f->vua, f->vva};
    a.fric = FricArgs{nx, ny, f->mask_u, f->mask_v, f->u1, f->v1, f->D_u, f->D_v, f->z0b_u, f->z0b_v, f->work_u,
                      f->work_v, f->ru, f->rv};
    a.spg = SpgArgs{nx, f->mask_u, f->mask_v, f->idx_u, f->idy_v, f->z, f->sp, f->H_t, f->D_t, Dmin, f->dpdx,
                    f->dpdy};
    a.taux = f->taux; a.tauy = f->tauy; a.tausx = f->tausx; a.tausy = f->tausy;
    int rc = getm_advection_2d_passes(uadv, ugrid, uugrid, uvgrid, uadv_ufirst, f->uua, f->uva, timestep, f->advD_u,
                                      f->D_uu, f->D_uv, f->advU, mixed != 0, &a.adv[0]);
    if (rc) return rc;
    rc = getm_advection_2d_passes(vadv, vgrid, vugrid, vvgrid, vadv_ufirst, f->vua, f->vva, timestep, f->advD_v,
                                  f->D_vu, f->D_vv, f->advV, mixed != 0, &a.adv[1]);
    if (rc) return rc;
    for (int d = 0; d < 2; d++)
        for (int s = 0; s < 2; s++)
            if (a.adv[d].pass[s].nx_ != nx || a.adv[d].pass[s].ny_ != ny) return GETM_ERR_ARG;
    a.Dsrc[0] = f->D_u; a.Dsrc[1] = f->D_v;
    a.advD[0] = f->advD_u; a.advD[1] = f->advD_v;
    a.advvar[0] = f->advU; a.advvar[1] = f->advV;
    a.Uo[0] = f->U; a.Uo[1] = f->V;
    a.sync = f->sync;
    return GETM_OK;
}

}  // namespace

// ---------------------------------------------------------------------------
// One substep of one domain: four launches
// ---------------------------------------------------------------------------
// What bounds these: on small planes the launches and one chain of latencies per
// kernel; on large ones instructions, L2 traffic (about 75 fields of a plane)
// and the FP64 pipe, which in the FP64 form is most of the time.  us per substep
// in a CUDA graph, one cooperative launch with six grid barriers -> the seven
// phases as seven launches -> these four:
//   mixed  64 x 64  45 -> 27 -> 20    200 x 150  46 -> 30 -> 28    400 x 300  56 -> 51 -> 46
//   FP64   64 x 64  56 -> 48 -> 26    150 x 120  58 -> 53 -> 36    220 x 160  68 -> 66 -> 52
// A barrier cost about 1.3 us and left every SM to the slowest block, and one
// register budget served all phases.  Each kernel but the first is launched
// when the blocks of the one before are done (programmatic dependent launch
// without an early trigger: blocks launched while the SMs are still busy land
// on whichever has room, and the FP64 pipes of those SMs then set the pace:
// FP64 220 x 160 57 -> 90 us; small planes of the mixed form, whose kernels
// leave SMs idle and wait for latencies, trigger as they begin: a 92 x 92
// member's step 948 -> 919 us, 184 x 184 1320 -> 1392) and waits for its end before
// it touches the fields; what precedes the first on the stream may be anything.
namespace {

constexpr int PH_XY = 2;  // rows of an x pass block

// Rows of a tile, chosen per plane (substep_rows): up to TR_MAX for the
// transports ((by + 1) x 33 staged points, one per thread) and DV_MAX for the
// depths ((by + 2) x 34).  Registers for two and three blocks of that size per SM.
constexpr int TR_MAX = 14, TR_THREADS = 512, DV_MAX = 9, DV_THREADS = 384;
static_assert((TR_MAX + 1) * 33 <= TR_THREADS && (DV_MAX + 2) * 34 <= DV_THREADS, "one staged point per thread");

// Waits for the kernel before; true when the error word is set (the kernel then leaves every field as it is).  The word is
// written only on the host's behalf, before the substep's first launch.
__device__ __forceinline__ bool substep_begin(const SubstepArgs& a)
{
    unsigned err = 0;
    if (a.sync) asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(err) : "l"(a.sync + 2) : "memory");
    if (a.early) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    return err != 0;
}

// The updated transports between the first two kernels: the momentum
// advections' scratch fields, free until the first advection pass.
__device__ __forceinline__ double* new_transport(const SubstepArgs& a, int d) { return a.adv[d].pass[0].fout[0]; }

// Phases 1 and 2: both transports into scratch (a neighbouring tile may still
// need the old ones), the Coriolis term of the second.  D1: the direction
// updated first; a tile of 32 x by points needs it on one more row and
// column, one point per thread; the second update's operands are loaded
// before the exchange.
template <bool MIXED, int D1>
__global__ void __launch_bounds__(TR_THREADS, 2)
    substep_transport_kernel(const __grid_constant__ SubstepArgs a, const int by)
{
    using C = typename std::conditional<MIXED, float, double>::type;
    constexpr int D2 = 1 - D1;
    constexpr int OX = D1 == 0 ? 1 : 0, OY = 1 - OX;  // columns west and rows south of the tile
    __shared__ double s1[TR_MAX + 1][33];
    const bool err = substep_begin(a);
    const int nx = a.nx, ny = a.ny, t = threadIdx.x;
    const int i0 = blockIdx.x * 32, j0 = blockIdx.y * by;
    auto interior = [&](int i, int j) {
        return i >= a.halox && i < nx - a.halox && j >= a.haloy && j < ny - a.haloy;
    };
    // the second direction's operands of the thread's point
    const int ty = t / 32, tx = t % 32, i = i0 + tx, j = j0 + ty;
    const bool own = ty < by && i < nx && j < ny;
    const int p = j * nx + i;
    TransportIn in2 = {};
    double cor2 = 0.0, f2 = 0.0, zp = 0.0;
    if (own) {
        in2 = transport_2d_load(a.tr[D2], p);
        f2 = a.corf[D2][p];
        zp = a.z[p];
    }
    // the first direction's staged point
    const int sj = t / 33, si = t - sj * 33, gi = i0 - OX + si, gj = j0 - OY + sj;
    if (sj <= by && gi >= 0 && gi < nx && gj >= 0 && gj < ny) {
        const int q = gj * nx + gi;
        const double cor = a.tr[D1].cor[q];
        const TransportIn in1 = transport_2d_load(a.tr[D1], q);
        s1[sj][si] = interior(gi, gj) ? transport_2d_value<MIXED>(in1, a.dt, cor) : in1.U;
    }
    __syncthreads();
    if (err || !own) return;
    new_transport(a, D1)[p] = s1[ty + OY][tx + OX];
    // U -> V with offsets (1, 0), negated; V -> U with offsets (0, 1)
    constexpr int ioff = D1 == 0 ? 1 : 0, joff = 1 - ioff;
    if (coriolis_2d_inside(nx, ny, ioff, joff, i, j)) {
        auto at = [&](int ai, int aj) { return s1[aj - j0 + OY][ai - i0 + OX]; };
        cor2 = coriolis_2d_value<C>(ioff, joff, i, j, at, f2, D1 == 0);
    } else {
        cor2 = coriolis_2d_outside<C>(a.cor_out[D2][p], f2, D1 == 0);
    }
    a.cor_out[D2][p] = cor2;
    new_transport(a, D2)[p] = interior(i, j) ? transport_2d_value<MIXED>(in2, a.dt, cor2) : in2.U;
    a.zo[p] = zp;
}

// Phases 3 to 5 on tiles of 32 x by points (T, U, V at (j, i) and X at
// (j, i) and (j + 1, i + 1)): new elevations of the tile and a point around
// it from the old ones (zo) and the new transports in scratch, the depths at
// T, U, V and X, and from them the velocities and the surface pressure
// gradient of the tile's points.  z, U and V are written, never read here.
// SPLIT where a block of DV_THREADS holds both halves (by <= 6): a 92 x 92 member's
// step 904 -> 810 us with the friction in blocks of its own; on larger planes one
// thread's two halves overlap better (mixed 400 x 300 47.9 us split, 46.5 not).
template <bool MIXED, bool SPLIT>
__global__ void __launch_bounds__(DV_THREADS, 3)
    substep_depth_kernel(const __grid_constant__ SubstepArgs a, const int by)
{
    using C = typename std::conditional<MIXED, float, double>::type;
    __shared__ double sz[DV_MAX + 2][34], szh[DV_MAX + 2][34];  // elevation: new, and the mean with the old
    __shared__ double sH[DV_MAX + 2][34], sD[DV_MAX + 2][34], sdh[DV_MAX + 2][34];  // T: H, D, D of the mean
    __shared__ double sB[DV_MAX + 2][34];                        // -H + Dmin
    __shared__ double sX[DV_MAX + 1][33], sU[DV_MAX + 1][33];    // X depths; sums of the means at i-1, i of row j-1
    const bool err = substep_begin(a);
    const DepthArgs& da = a.depth;
    const int nx = a.nx, ny = a.ny, t = threadIdx.x;
    const int i0 = blockIdx.x * 32, j0 = blockIdx.y * by;
    const double* __restrict__ Us = new_transport(a, 0);
    const double* __restrict__ Vs = new_transport(a, 1);
    // SPLIT: the first 32 by threads take the U halves of the points, the next the V
    // halves (small planes, where one thread's chain of instructions is the
    // time); else one thread takes both.  The operands of the thread's point and
    // of its X point are loaded while the elevations are staged
    const int npt = 32 * by, w = SPLIT && t >= npt ? t - npt : t;
    const int ty = w / 32, tx = w % 32, i = i0 + tx, j = j0 + ty;
    const bool own = w < npt && i < nx && j < ny;
    const bool east = i < nx - 1, north = j < ny - 1;
    const int p = j * nx + i;
    struct Half {
        int m;
        double H, T, Te, Tn;
    };
    auto load = [&](int h) {
        Half o{0, 0.0, 0.0, 0.0, 0.0};
        if (own) {
            const double* __restrict__ Ts = h == 0 ? Us : Vs;
            o.m = (h == 0 ? da.mU : da.mV)[p];
            o.H = (h == 0 ? da.HU : da.HV)[p];
            o.T = Ts[p];
            if (east) o.Te = Ts[p + 1];
            if (north) o.Tn = Ts[p + nx];
        }
        return o;
    };
    Half o0, o1;
    if constexpr (SPLIT) {
        o0 = load(t < npt ? 0 : 1);
    } else {
        o0 = load(0);
        o1 = load(1);
    }
    const int xj = t / 33, xi = t - xj * 33, Xj = j0 + xj, Xi = i0 + xi;
    const bool xin = xj <= by && Xi <= nx && Xj <= ny;
    const int px = Xj * (nx + 1) + Xi;
    int mX = 0;
    double HX = 0.0;
    if (xin) { mX = da.mX[px]; HX = da.HX[px]; }

    // elevation (simulation.py:1468-1486) and T depths of the staged point
    const int sj = t / 34, si = t - sj * 34, gi = i0 - 1 + si, gj = j0 - 1 + sj;
    if (sj < by + 2) {
        double z = 0.0, zh = 0.0, D = 0.0, H = 0.0, dh = 0.0, B = 0.0;
        if (gi >= 0 && gi < nx && gj >= 0 && gj < ny) {
            const int g = gj * nx + gi;
            const int m = a.mT[g];
            const double zo = a.zo[g];
            H = da.HT[g];
            B = -H + da.Dmin;
            z = zo;
            if (gi >= a.halox && gi < nx - a.halox && gj >= a.haloy && gj < ny - a.haloy) {
                const double Uw = Us[g - 1], dyw = a.dyU[g - 1], Uc = Us[g], dye = a.dyU[g];
                const double Vs0 = Vs[g - nx], dxs = a.dxV[g - nx], Vc = Vs[g], dxn = a.dxV[g];
                const double ia = a.iareaT[g], fw = a.fwf[g];
                if (m == 1) z = elevation_new(zo, a.dt, Uw, dyw, Uc, dye, Vs0, dxs, Vc, dxn, ia, fw);
            }
            zh = getm_half(zo + z);
            D = m != 0 ? getm_fmax_i(H + z, -1000.0) : da.DT[g];
            dh = m != 0 ? getm_fmax_i(H + zh, da.Dmin) : zh;
            if (!err && sj >= 1 && sj <= by && si >= 1 && si <= 32) {  // the tile's own point
                if (m == 1) a.z[g] = z;
                if (m != 0) da.DT[g] = D;
                da.DclipT[g] = dclamp_min(D, da.Dmin);
                da.workT[g] = dh;
            }
        }
        sz[sj][si] = z; szh[sj][si] = zh; sH[sj][si] = H; sD[sj][si] = D; sdh[sj][si] = dh; sB[sj][si] = B;
    }
    __syncthreads();
    if (err) return;
    // X depths: interp_xy T->X (offsets 1, 1) where it writes, else the
    // previous X._work value
    if (xin) {
        const bool mine = xj < by && xi < 32;
        const double south = szh[xj][xi] + szh[xj][xi + 1];  // (also z_U of the point south-west)
        sU[xj][xi] = south;
        double zx;
        if (Xj >= 1 && Xj <= ny - 1 && Xi >= 1 && Xi <= nx - 1) {
            zx = getm_quarter(south + szh[xj + 1][xi] + szh[xj + 1][xi + 1]);
            if (mine) da.workX[px] = zx;
        } else {
            zx = da.workX[px];
        }
        const double dx = mX != 0 ? getm_fmax_i(HX + zx, da.Dmin) : da.DX[px];
        if (mine && mX != 0) da.DX[px] = dx;
        sX[xj][xi] = dx;
    }
    __syncthreads();
    const double twoDmin = 2 * da.Dmin;
    const float twoDmin_f = 2.f * getm_d2f_approx(da.Dmin), ialpha_f = getm_d2f_approx(da.ialpha);
    if (!own) return;
    auto half = [&](int h, const Half& o) {
        const int y = ty + 1, x = tx + 1;  // the point in the staged tile
        // z_U = interp_x(z_T_half, ioffset 0) for i < nx-1, z_V = interp_y for
        // j < ny-1, else the old value
        double* work = h == 0 ? da.workU : da.workV;
        double* Dp = h == 0 ? da.DU : da.DV;
        double z, D;
        if (h == 0 ? east : north) {
            z = getm_half(h == 0 ? sU[y][x] : szh[y][x] + szh[y + 1][x]);
            work[p] = z;
        } else {
            z = work[p];
        }
        if (o.m != 0) {
            D = getm_fmax_i(o.H + z, da.Dmin);
            Dp[p] = D;
            (h == 0 ? da.alphaU : da.alphaV)[p] =
                MIXED ? alpha_of_f(D, twoDmin_f, ialpha_f) : alpha_of(D, twoDmin, da.ialpha);
        } else {
            D = Dp[p];
        }
        a.advD[h][p] = D;
        // UU.D[:, :-1] = D_T_half[:, 1:], VV.D[:-1, :] = D_T_half[1:, :], UV.D = VU.D = X.D[1:, 1:]
        const double Dx = sX[ty + 1][tx + 1];
        double Dt;
        if (h == 0) {
            Dt = east ? sdh[y][x + 1] : da.DUU[p];
            if (east) da.DUU[p] = Dt;
            da.DUV[p] = Dx;
        } else {
            Dt = north ? sdh[y + 1][x] : da.DVV[p];
            if (north) da.DVV[p] = Dt;
            da.DVU[p] = Dx;
        }
        momentum_2d_velocities_half<C>(a.vel, h, p, east, north, o.T, o.Te, o.Tn, D, h == 0 ? Dt : Dx, h == 0 ? Dx : Dt);
        // the transport's final value, and what only reads it
        a.tr[h].U[p] = o.T;
        if (a.accumulate) {
            double* cum = h == 0 ? a.Ucum : a.Vcum;
            cum[p] = cum[p] + o.T;
        }
        if (h == 0) {
            coriolis_from<C>(a, a.ufirst ? 1 : 0, i, j, a.ufirst ? Vs : Us);
            if (east) interp_pair_point<double>(a.taux, a.tausx, p, 1, 0);
        } else if (north) {
            interp_pair_point<double>(a.tauy, a.tausy, p, nx, 0);
        }
        if (i >= a.halox && i < nx - a.halox && j >= a.haloy && j < ny - a.haloy) {
            const int dx = h == 0 ? 1 : 0, dy = 1 - dx;
            spg_half<MIXED>(h == 0 ? a.spg.dpdx : a.spg.dpdy, a.spg.Dmin, p, o.m, sz[y][x], sz[y + dy][x + dx], sH[y][x],
                            sH[y + dy][x + dx], sD[y][x], sD[y + dy][x + dx], sB[y][x], sB[y + dy][x + dx], a.spg.sp[p],
                            a.spg.sp[p + (h == 0 ? 1 : nx)], (h == 0 ? a.spg.idxu : a.spg.idyv)[p]);
        }
    };
    if constexpr (SPLIT) {
        half(t < npt ? 0 : 1, o0);
    } else {
        half(0, o0);
        half(1, o1);
    }
}

// Phases 6 and 7: advection pass PASS in direction DIR of U (block z 0; d0 =
// 0) and V, nd of them.  With the first pass, the blocks share out the friction
// of their direction's equation and fwf = pe (which phase 3 still needed): the
// FP64 form's friction takes as long as its pass, so every block gets its part.
// On small planes (early) blocks of their own, z >= nd, take it instead.
template <bool MIXED, int PASS, int DIR, int BY>
__global__ void __launch_bounds__(32 * BY)
    substep_advection_kernel(const __grid_constant__ SubstepArgs a, int d0, int nd)
{
    using C = typename std::conditional<MIXED, float, double>::type;
    if (substep_begin(a)) return;
    const int tx = threadIdx.x, ty = threadIdx.y;
    const bool apart = blockIdx.z >= nd;
    const int d = d0 + (apart ? blockIdx.z - nd : blockIdx.z);
    const HPassArgs<double>& pa = a.adv[d].pass[PASS];
    if (PASS == 0 && (apart || gridDim.z == nd)) {
        const int n = a.nx * a.ny, step = 32 * BY * gridDim.x * gridDim.y;
        for (int p = ((blockIdx.y * gridDim.x + blockIdx.x) * BY + ty) * 32 + tx; p < n; p += step) {
            if (d == 0) a.fwf[p] = a.pe[p];
            if (a.friction) momentum_2d_friction_half<C>(a.fric, d, p % a.nx, p / a.nx);
        }
    }
    if (apart) return;
    if (PASS == 1 && d == 0 && blockIdx.x == 0 && blockIdx.y == 0 && tx == 0 && ty == 0 && a.time)
        *a.time = *a.time + a.dt;
    auto pass = [&](const auto& epi) {
        using E = typename std::decay<decltype(epi)>::type;
        if constexpr (DIR == 1) {
            const int row = blockIdx.y * BY + ty;
            if (row < pa.ny_) hpass_x_inc_body<double, E, double, C>(pa, blockIdx.x, row, tx, epi);
        } else {
            __shared__ YIncSmem<double, C, BY> sm;
            hpass_y_inc_body<double, E, double, C, BY>(pa, blockIdx.x, blockIdx.y, 0, tx, ty, sm, epi);
        }
    };
    if constexpr (PASS == 1) pass(ReconstructEpi{a.advvar[d], a.Uo[d], a.idt, a.haloy, a.ny - a.haloy - 1});
    else pass(NoEpi());
}

template <typename K, typename... A>
int launch_substep(K kernel, dim3 grid, dim3 block, bool first, cudaStream_t stream, const A&... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = first ? 0 : 1;
    if (cudaLaunchKernelEx(&cfg, kernel, args...) != cudaSuccess) return GETM_ERR_CUDA;
    GETM_CHECK_LAUNCH();
    return GETM_OK;
}

// One launch for both directions' pass where they share the axis (they do
// unless the host gave the two advections different orders)
template <bool MIXED, int PASS>
int launch_substep_advection(const SubstepArgs& a, cudaStream_t stream, bool first = false)
{
    const bool one = a.adv[0].dir[PASS] == a.adv[1].dir[PASS];
    const int nd = one ? 2 : 1, nz = PASS == 0 && a.early ? 2 * nd : nd;
    for (int d = 0; d < 3 - nd; d++) {
        int rc;
        if (a.adv[d].dir[PASS] == 1) {
            const dim3 g(div_up(a.nx + 1, HX_STRIDE), div_up(a.ny, PH_XY), nz);
            rc = launch_substep(substep_advection_kernel<MIXED, PASS, 1, PH_XY>, g, dim3(32, PH_XY), first && d == 0,
                                stream, a, d, nd);
        } else {
            const int by = MIXED ? 4 : hpass_y_rows((long long)div_up(a.nx, 32) * nd, a.ny, true);
            const dim3 g(div_up(a.nx, 32), div_up(a.ny + 1, by - 1), nz), b(32, by);
            const bool f = first && d == 0;
            if (by == 4)
                rc = launch_substep(substep_advection_kernel<MIXED, PASS, 2, 4>, g, b, f, stream, a, d, nd);
            else
                rc = launch_substep(substep_advection_kernel<false, PASS, 2, 16>, g, b, f, stream, a, d, nd);
        }
        if (rc) return rc;
    }
    return GETM_OK;
}

// Rows of a tile with `edge` more staged: the height up to `most` that leaves
// the SM with most tiles the fewest staged rows.  A plane then goes in one
// wave where it can (400 x 300: 442 depth tiles of 9 rows on 152 SMs of three),
// and a small one spreads over as many SMs as it can, whose FP64 pipes it waits
// for (mixed form: four rows at least, as more blocks only add edges: a 92 x 92
// member's step 948 us, with two rows 954).
inline int substep_rows(int nx, int ny, int most, int edge, int least_rows)
{
    int best = most;
    long long least = 0;
    for (int by = most; by >= least_rows; by--) {
        const long long tiles = (long long)div_up(nx, 32) * div_up(ny, by);
        const long long load = (tiles + GETM_SMS - 1) / GETM_SMS * (by + edge);
        if (by == most || load < least) { least = load; best = by; }
    }
    return best;
}

template <bool MIXED>
int launch_substep_kernels(const SubstepArgs& a, cudaStream_t stream)
{
    const int tr = substep_rows(a.nx, a.ny, TR_MAX, 1, MIXED ? 4 : 2);
    const int dv = substep_rows(a.nx + 1, a.ny + 1, DV_MAX, 2, MIXED ? 4 : 2);
    const dim3 tg(div_up(a.nx, 32), div_up(a.ny, tr)), tb(div_up((tr + 1) * 33, 32) * 32);
    const bool split = 64 * dv <= DV_THREADS;
    const int dt = div_up((dv + 2) * 34, 32) * 32;
    const dim3 dg(div_up(a.nx + 1, 32), div_up(a.ny + 1, dv)), db(split ? std::max(dt, 64 * dv) : dt);
    int rc = a.ufirst ? launch_substep(substep_transport_kernel<MIXED, 0>, tg, tb, true, stream, a, tr)
                      : launch_substep(substep_transport_kernel<MIXED, 1>, tg, tb, true, stream, a, tr);
    if (!rc) rc = split ? launch_substep(substep_depth_kernel<MIXED, true>, dg, db, false, stream, a, dv)
                        : launch_substep(substep_depth_kernel<MIXED, false>, dg, db, false, stream, a, dv);
    if (!rc) rc = launch_substep_advection<MIXED, 0>(a, stream);
    if (!rc) rc = launch_substep_advection<MIXED, 1>(a, stream);
    return rc;
}

}  // namespace

extern "C" int getm_split2d_substep(const getm_split2d_fields* f, int nx, int ny, int halox, int haloy, int mixed,
                                    int ufirst, int accumulate, int friction, double timestep, double Dmin,
                                    double Dcrit, getm_advection* uadv, getm_grid* ugrid, getm_grid* uugrid,
                                    getm_grid* uvgrid, int uadv_ufirst, getm_advection* vadv, getm_grid* vgrid,
                                    getm_grid* vugrid, getm_grid* vvgrid, int vadv_ufirst, cudaStream_t stream)
{
    SubstepArgs a;
    int rc = substep_args(a, f, nx, ny, halox, haloy, mixed, ufirst, accumulate, friction, timestep, Dmin, Dcrit,
                          uadv, ugrid, uugrid, uvgrid, uadv_ufirst, vadv, vgrid, vugrid, vvgrid, vadv_ufirst);
    if (rc) return rc;
    // (see above: mixed form, depth tiles of four rows for at most every SM)
    a.early = mixed && (long long)div_up(nx + 1, 32) * div_up(ny + 1, 4) <= GETM_SMS;
    return mixed ? launch_substep_kernels<true>(a, stream) : launch_substep_kernels<false>(a, stream);
}

// ---------------------------------------------------------------------------
// Some phases of a substep, one launch each
// ---------------------------------------------------------------------------
// For a substep with work between its phases: the 3D step between the elevation
// and the depths, the open boundaries' mirrored transports, depths and
// elevations.  One by one its operations are nineteen launches.
namespace {

constexpr int PH_PY = 4;  // rows of a block

template <bool MIXED, int PH>
__global__ void __launch_bounds__(32 * PH_PY) phase_points_kernel(const __grid_constant__ SubstepArgs a, int spg)
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int i = blockIdx.x * 32 + threadIdx.x, j = blockIdx.y * PH_PY + threadIdx.y;
    if (i < a.nx && j < a.ny) phase_point<MIXED>(a, PH, a.ufirst ? 0 : 1, i, j, j * a.nx + i, spg != 0);
}

template <bool MIXED>
__global__ void __launch_bounds__(32 * PH_PY) phase_depth_kernel(const __grid_constant__ SubstepArgs a)
{
    __shared__ double szh[PH_PY + 2][UD_BX + 2];
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int i = blockIdx.x * 32 + threadIdx.x, j = blockIdx.y * PH_PY + threadIdx.y;
    if (i < a.nx && j < a.ny) phase_point<MIXED>(a, 3, 0, i, j, j * a.nx + i);
    update_depth_2d_tile<PH_PY, MIXED>(a.depth, blockIdx.x, blockIdx.y, threadIdx.x, threadIdx.y, szh);
}

template <bool MIXED>
int launch_phases(const SubstepArgs& a, int first, int last, int spg, cudaStream_t stream)
{
    const dim3 b(32, PH_PY), g(div_up(a.nx, 32), div_up(a.ny, PH_PY));
    const dim3 gd(div_up(a.nx + 1, UD_BX), div_up(a.ny + 1, PH_PY));
    for (int ph = first; ph <= last; ph++) {
        const bool f = ph == first;
        int rc;
        switch (ph) {
        case 1: rc = launch_substep(phase_points_kernel<MIXED, 0>, g, b, f, stream, a, spg); break;
        case 2: rc = launch_substep(phase_points_kernel<MIXED, 1>, g, b, f, stream, a, spg); break;
        case 3: rc = launch_substep(phase_points_kernel<MIXED, 2>, g, b, f, stream, a, spg); break;
        case 4: rc = launch_substep(phase_depth_kernel<MIXED>, gd, b, f, stream, a); break;
        case 5: rc = launch_substep(phase_points_kernel<MIXED, 4>, g, b, f, stream, a, spg); break;
        case 6: rc = launch_substep_advection<MIXED, 0>(a, stream, f); break;
        default: rc = launch_substep_advection<MIXED, 1>(a, stream, f); break;
        }
        if (rc) return rc;
    }
    return GETM_OK;
}

}  // namespace

extern "C" int getm_split2d_phases(const getm_split2d_fields* f, int nx, int ny, int halox, int haloy, int mixed,
                                   int ufirst, int accumulate, int friction, double timestep, double Dmin,
                                   double Dcrit, getm_advection* uadv, getm_grid* ugrid, getm_grid* uugrid,
                                   getm_grid* uvgrid, int uadv_ufirst, getm_advection* vadv, getm_grid* vgrid,
                                   getm_grid* vugrid, getm_grid* vvgrid, int vadv_ufirst, int first, int last,
                                   int spg, cudaStream_t stream)
{
    if (first < 1 || last < first || last > 7) return GETM_ERR_ARG;
    SubstepArgs a;
    int rc = substep_args(a, f, nx, ny, halox, haloy, mixed, ufirst, accumulate, friction, timestep, Dmin, Dcrit,
                          uadv, ugrid, uugrid, uvgrid, uadv_ufirst, vadv, vgrid, vugrid, vvgrid, vadv_ufirst);
    if (rc) return rc;
    a.sync = nullptr;  // (the error word concerns whole substeps)
    return mixed ? launch_phases<true>(a, first, last, spg, stream) : launch_phases<false>(a, first, last, spg, stream);
}

// ---------------------------------------------------------------------------
// Substeps of many independent domains in one launch
// ---------------------------------------------------------------------------
// An ensemble of domains of uneven size (ensemble members, served requests)
// advances each member by `split` substeps per 3D step, the last of which
// runs the member's 3D step.  The other substeps of every member run here as
// one cooperative launch per substep index k: launch k advances every member
// with more than k such substeps by one substep.  The seven phases and their
// device functions are those of the single substep; within a phase the blocks
// walk one list of block-sized work items spanning all members (512-point
// chunks, depth tiles, advection row groups or tiles), so the small planes
// of many members fill the GPU together and one set of grid barriers serves
// them all.  Members are sorted by their number of substeps (descending), so
// the members of launch k are a prefix of the table and each phase's items
// are a prefix of its offset list.  Each member keeps its own arguments, time
// step and transport order: its order at launch k of a round is its recorded
// order flipped (k + round_parity * split) times.
namespace {

constexpr int SB_PHASES = 7;

struct BatchMember {
    SubstepArgs a;
    int nsub;              // substeps without 3D step per round: takes part in launches k < nsub
    int split;             // substeps per round
    int n;                 // points nx * ny
    int pts;               // block items of a point phase
    int dtiles, dntx;      // depth tiles, and their count along x
    int adv_items[2][2];   // [U/V][pass] block items
    int adv_nbx[2][2];     // [U/V][pass] row segments (x pass) or tile columns (y pass)
};

// Block items of one momentum advection pass over the plane.
template <bool MIXED>
void pass_items(const HPassArgs<double>& pa, int dir, int& items, int& nbx)
{
    if (dir == 1) {
        nbx = div_up(pa.nx_ + 1, HX_STRIDE);
        items = nbx * div_up(pa.ny_, SS_BY);
    } else {
        nbx = div_up(pa.nx_, 32);
        const int nby = div_up(pa.ny_ + 1, HY_STRIDE);
        items = nbx * nby;
    }
}

// Items of each phase for one member (the order within a phase is fixed
// below in batch_item).
void phase_items(const BatchMember& m, int out[SB_PHASES])
{
    out[0] = out[1] = out[2] = out[4] = m.pts;
    out[3] = m.dtiles + m.pts;
    out[5] = (m.a.friction ? m.pts : 0) + m.adv_items[0][0] + m.adv_items[1][0];
    out[6] = m.adv_items[0][1] + m.adv_items[1][1];
}

// Block item q of one pass of the momentum advection.
template <bool MIXED, typename Epi = NoEpi>
__device__ __forceinline__ void batch_pass_item(const HPassArgs<double>& pa, int dir, int nbx, int q, SubstepSmem& sm,
                                                int tx, int ty, const Epi& epi = Epi())
{
    using C = typename std::conditional<MIXED, float, double>::type;
    if (dir == 1) {
        const long long row = (long long)(q / nbx) * SS_BY + ty;
        if (row < pa.ny_) hpass_x_inc_body<double, Epi, double, C>(pa, q % nbx, row, tx, epi);
    } else {
        if constexpr (MIXED) hpass_y_inc_body<double, Epi, double, float>(pa, q % nbx, q / nbx, 0, tx, ty, sm.yf, epi);
        else hpass_y_inc_body<double, Epi, double, double>(pa, q % nbx, q / nbx, 0, tx, ty, sm.yd, epi);
        __syncthreads();  // shared memory is reused by the block's next item
    }
}

// Work item q of phase ph of one member: the same operations, in the same
// order per point, as the phases listed at the top.
template <bool MIXED>
__device__ void batch_item(const BatchMember& m, int ph, int q, int ufirst, SubstepSmem& sm, int tx, int ty)
{
    const SubstepArgs& a = m.a;
    const int nx = a.nx, ny = a.ny;
    const int jlo = a.haloy, jhi = ny - a.haloy - 1;
    const int d1 = ufirst ? 0 : 1;
    auto points = [&](int php, int qq) {
        const int p = qq * SS_THREADS + ty * 32 + tx;
        if (p < m.n) phase_point<MIXED>(a, php, d1, p % nx, p / nx, p);
    };
    switch (ph) {
    case 0:
        points(0, q);
        break;
    case 1:
        points(1, q);
        break;
    case 2:
        points(2, q);
        break;
    case 3:
        if (q < m.dtiles) {
            update_depth_2d_tile<SS_BY, MIXED>(a.depth, q % m.dntx, q / m.dntx, tx, ty, sm.szh);
            __syncthreads();
        } else {
            points(3, q - m.dtiles);
        }
        break;
    case 4:
        points(4, q);
        break;
    case 5: {
        int r = q;
        if (a.friction) {
            if (r < m.pts) {
                points(5, r);
                break;
            }
            r -= m.pts;
        }
        if (r < m.adv_items[0][0]) {
            batch_pass_item<MIXED>(a.adv[0].pass[0], a.adv[0].dir[0], m.adv_nbx[0][0], r, sm, tx, ty);
            break;
        }
        r -= m.adv_items[0][0];
        batch_pass_item<MIXED>(a.adv[1].pass[0], a.adv[1].dir[0], m.adv_nbx[1][0], r, sm, tx, ty);
        break;
    }
    default: {
        // the model time moves on once per member, in its first item of the
        // last phase (after the last barrier)
        if (q == 0 && tx == 0 && ty == 0 && a.time) *a.time = *a.time + a.dt;
        const int d = q < m.adv_items[0][1] ? 0 : 1;
        const int r = d == 0 ? q : q - m.adv_items[0][1];
        const ReconstructEpi epi{a.advvar[d], a.Uo[d], a.idt, jlo, jhi};
        batch_pass_item<MIXED>(a.adv[d].pass[1], a.adv[d].dir[1], m.adv_nbx[d][1], r, sm, tx, ty, epi);
        break;
    }
    }
}

// off: SB_PHASES lists of nmember + 1 item offsets (phase-major).
template <bool MIXED>
__global__ void __launch_bounds__(SS_THREADS, MIXED ? 2 : 1)
    substep_batch_kernel(const BatchMember* __restrict__ mem, const int* __restrict__ off, int nmember, int P,
                         int k, int round_parity, unsigned* sync)
{
    __shared__ SubstepSmem sm;
    __shared__ int s_ok;
    const int tx = threadIdx.x, ty = threadIdx.y;
    unsigned target = 0;
    if (tx == 0 && ty == 0) s_ok = ld_acquire(&sync[2]) == 0;
    __syncthreads();
    if (!s_ok) return;
    for (int ph = 0; ph < SB_PHASES; ph++) {
        const int* o = off + ph * (nmember + 1);
        const int total = o[P];
        for (int w = blockIdx.x; w < total; w += gridDim.x) {
            // the member of item w: the last m < P with o[m] <= w
            int lo = 0, hi = P - 1;
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (o[mid] <= w) lo = mid;
                else hi = mid - 1;
            }
            const BatchMember& m = mem[lo];
            const int ufirst = m.a.ufirst ^ ((k + round_parity * m.split) & 1);
            batch_item<MIXED>(m, ph, w - o[lo], ufirst, sm, tx, ty);
        }
        if (ph + 1 < SB_PHASES && !grid_barrier(sync, target, s_ok)) return grid_exit(sync);
    }
    grid_exit(sync);
}

template <bool MIXED>
int batch_blocks(int dev, int* blocks)
{
    static int cache[SS_MAX_DEVICES];
    static std::mutex mutex;
    if (dev < 0 || dev >= SS_MAX_DEVICES) return GETM_ERR_ARG;
    std::lock_guard<std::mutex> lock(mutex);
    if (cache[dev] == 0) {
        int sms = 0, coop = 0, per_sm = 0;
        if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop)
            return GETM_ERR_CUDA;
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return GETM_ERR_CUDA;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, substep_batch_kernel<MIXED>, SS_THREADS, 0) !=
                cudaSuccess ||
            per_sm < 1)
            return GETM_ERR_CUDA;
        cache[dev] = sms * per_sm;
    }
    *blocks = cache[dev];
    return GETM_OK;
}

}  // namespace

struct getm_substep_batch {
    int nmember, mixed;
    BatchMember* host;      // as set, in member order
    int* set;               // which members were set
    int* order;             // sorted position -> member index
    int* nsub_sorted;       // nsub of the sorted members
    BatchMember* dmem;      // device table (sorted)
    int* doff;              // device offsets
};

extern "C" int getm_substep_batch_create(int nmember, int mixed, getm_substep_batch** out)
{
    if (!out || nmember < 1) return GETM_ERR_ARG;
    getm_substep_batch* b = (getm_substep_batch*)calloc(1, sizeof(getm_substep_batch));
    if (!b) return GETM_ERR_ALLOC;
    b->nmember = nmember;
    b->mixed = mixed != 0;
    b->host = (BatchMember*)calloc(nmember, sizeof(BatchMember));
    b->set = (int*)calloc(nmember, sizeof(int));
    b->order = (int*)calloc(nmember, sizeof(int));
    b->nsub_sorted = (int*)calloc(nmember, sizeof(int));
    if (!b->host || !b->set || !b->order || !b->nsub_sorted) {
        free(b->host); free(b->set); free(b->order); free(b->nsub_sorted); free(b);
        return GETM_ERR_ALLOC;
    }
    *out = b;
    return GETM_OK;
}

extern "C" int getm_substep_batch_finalize(getm_substep_batch* b)
{
    if (!b) return GETM_OK;
    cudaFree(b->dmem);
    cudaFree(b->doff);
    free(b->host); free(b->set); free(b->order); free(b->nsub_sorted);
    free(b);
    return GETM_OK;
}

extern "C" int getm_substep_batch_set(getm_substep_batch* b, int member, int nsub, int split,
                                      const getm_split2d_fields* f, int nx, int ny, int halox, int haloy, int ufirst,
                                      int accumulate, int friction, double timestep, double Dmin, double Dcrit,
                                      getm_advection* uadv, getm_grid* ugrid, getm_grid* uugrid, getm_grid* uvgrid,
                                      int uadv_ufirst, getm_advection* vadv, getm_grid* vgrid, getm_grid* vugrid,
                                      getm_grid* vvgrid, int vadv_ufirst)
{
    if (!b || member < 0 || member >= b->nmember || nsub < 0 || split < nsub + 1 || b->dmem) return GETM_ERR_ARG;
    BatchMember& m = b->host[member];
    int rc = substep_args(m.a, f, nx, ny, halox, haloy, b->mixed, ufirst, accumulate, friction, timestep, Dmin,
                          Dcrit, uadv, ugrid, uugrid, uvgrid, uadv_ufirst, vadv, vgrid, vugrid, vvgrid, vadv_ufirst);
    if (rc) return rc;
    m.a.sync = nullptr;  // the batch launch has its own barrier words
    m.nsub = nsub;
    m.split = split;
    m.n = nx * ny;
    m.pts = div_up(m.n, SS_THREADS);
    m.dntx = div_up(nx + 1, UD_BX);
    m.dtiles = m.dntx * div_up(ny + 1, SS_BY);
    for (int d = 0; d < 2; d++)
        for (int s = 0; s < 2; s++) {
            if (b->mixed) pass_items<true>(m.a.adv[d].pass[s], m.a.adv[d].dir[s], m.adv_items[d][s], m.adv_nbx[d][s]);
            else pass_items<false>(m.a.adv[d].pass[s], m.a.adv[d].dir[s], m.adv_items[d][s], m.adv_nbx[d][s]);
        }
    b->set[member] = 1;
    return GETM_OK;
}

extern "C" int getm_substep_batch_upload(getm_substep_batch* b)
{
    if (!b || b->dmem) return GETM_ERR_ARG;
    const int n = b->nmember;
    for (int q = 0; q < n; q++)
        if (!b->set[q]) return GETM_ERR_ARG;
    // members by their substep count, descending (stable)
    for (int q = 0; q < n; q++) b->order[q] = q;
    for (int q = 1; q < n; q++) {
        const int x = b->order[q];
        int r = q;
        while (r > 0 && b->host[b->order[r - 1]].nsub < b->host[x].nsub) {
            b->order[r] = b->order[r - 1];
            r--;
        }
        b->order[r] = x;
    }
    BatchMember* sorted = (BatchMember*)malloc(sizeof(BatchMember) * n);
    int* off = (int*)calloc((size_t)SB_PHASES * (n + 1), sizeof(int));
    if (!sorted || !off) { free(sorted); free(off); return GETM_ERR_ALLOC; }
    long long total[SB_PHASES] = {0};
    for (int q = 0; q < n; q++) {
        sorted[q] = b->host[b->order[q]];
        b->nsub_sorted[q] = sorted[q].nsub;
        int it[SB_PHASES];
        phase_items(sorted[q], it);
        for (int ph = 0; ph < SB_PHASES; ph++) {
            total[ph] += it[ph];
            off[ph * (n + 1) + q + 1] = (int)total[ph];
        }
    }
    int rc = GETM_OK;
    for (int ph = 0; ph < SB_PHASES; ph++)
        if (total[ph] >= (1ll << 31)) rc = GETM_ERR_ARG;
    if (!rc && (cudaMalloc(&b->dmem, sizeof(BatchMember) * n) != cudaSuccess ||
                cudaMalloc(&b->doff, sizeof(int) * SB_PHASES * (n + 1)) != cudaSuccess))
        rc = GETM_ERR_ALLOC;
    if (!rc && (cudaMemcpy(b->dmem, sorted, sizeof(BatchMember) * n, cudaMemcpyHostToDevice) != cudaSuccess ||
                cudaMemcpy(b->doff, off, sizeof(int) * SB_PHASES * (n + 1), cudaMemcpyHostToDevice) != cudaSuccess))
        rc = GETM_ERR_CUDA;
    free(sorted);
    free(off);
    if (rc) {
        cudaFree(b->dmem); cudaFree(b->doff);
        b->dmem = nullptr; b->doff = nullptr;
    }
    return rc;
}

extern "C" int getm_substep_batch_participants(const getm_substep_batch* b, int k, int* count)
{
    if (!b || !count || k < 0) return GETM_ERR_ARG;
    int P = 0;
    while (P < b->nmember && b->nsub_sorted[P] > k) P++;
    *count = P;
    return GETM_OK;
}

extern "C" int getm_substep_batch_launch(getm_substep_batch* b, int k, int round_parity, unsigned int* sync,
                                         cudaStream_t stream)
{
    if (!b || !b->dmem || !sync || k < 0 || round_parity < 0 || round_parity > 1) return GETM_ERR_ARG;
    int P = 0;
    getm_substep_batch_participants(b, k, &P);
    if (P == 0) return GETM_OK;
    int dev = 0, blocks = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return GETM_ERR_CUDA;
    int rc = b->mixed ? batch_blocks<true>(dev, &blocks) : batch_blocks<false>(dev, &blocks);
    if (rc) return rc;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(32, SS_BY);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const BatchMember* mem = b->dmem;
    const int* off = b->doff;
    const int n = b->nmember;
    cudaError_t e = b->mixed ? cudaLaunchKernelEx(&cfg, substep_batch_kernel<true>, mem, off, n, P, k, round_parity, sync)
                             : cudaLaunchKernelEx(&cfg, substep_batch_kernel<false>, mem, off, n, P, k, round_parity,
                                                  sync);
    if (e != cudaSuccess) return GETM_ERR_CUDA;
    GETM_CHECK_LAUNCH();
    return GETM_OK;
}
