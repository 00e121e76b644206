// mgp_kernels.cuh -- kernel launchers shared by the host drivers (mgp_host.cu)
// and the kernels (mgp_kernels.cu).
#pragma once
#include <cuda.h>

#include "mgp_core.cuh"

namespace mgp {

// Most blocks a reduction uses (4 per SM of a B200): launch_reduce's partials
// take two doubles per block.
constexpr int kRedBlocksMax = 592;

// Reduction kinds of launch_reduce.
enum RedKind { RED_SUMSQ = 0, RED_MAXABS = 1, RED_DOT = 2, RED_JSUM = 3, RED_ABSSUM = 4 };

// Values of a solver's device status word.  A kernel records the first error
// it meets and never overwrites one already there (set_status), so the host
// sees the cause, not a later consequence.
enum DevStatus {
    DST_OK = 0,
    DST_TIMEOUT = 2,      // a bounded device wait (tile loads, grid barrier) ran out
    DST_NONFINITE = 3,    // a non-finite residual in a device-side solve (bottom BiCGStab)
};
#ifdef __CUDACC__
__device__ __forceinline__ void set_status(int* s, int v) {
    if (s && v) atomicCAS(s, 0, v);
}
#endif

// A grid barrier gives up after this long by default (%globaltimer
// nanoseconds): far above any real wait between two barriers of the coarse
// cycle (milliseconds at most).
constexpr unsigned long long kGridWaitNsDefault = 1000000000ull;

// Barrier and reduction partials of a cooperative grid running the
// coarse cycle (k_coarse_cycle_grid).
struct GridCtl {
    unsigned* bar;   // [0] arrivals, [1] generation; arrivals 0 at launch
    double* part;    // 2 x (CTAs) partial sums
    int* status;     // DST_TIMEOUT if a barrier wait gives up; once nonzero, barriers stop waiting
    unsigned long long wait_ns;   // a CTA's longest wait at one barrier
};

// Levels of at most this many cells run as dense operators in the staged coarse
// cycle (TinyLv), where every side is Dirichlet, Neumann or periodic.
constexpr int kTinyCells = 64;
// A level's smoothing sweep, operator and bottom preconditioner as dense
// matrices over its n cells (i fastest), stored by input: entry (k, m) at
// [m * n + k].  A sweep and the operator read up to four stored Neumann ghosts
// (where a Dirichlet or periodic x side meets a Neumann y side, or the other way
// round, the corner cell's closure does): inputs n .. n + ng - 1.
enum { TM_U, TM_S, TM_A, TM_M, TM_AM, TM_C, kTinyMats };
struct TinyLv {
    int n;               // cells, 0: not a tiny level
    int ng;              // stored ghosts that enter U and A
    int gi[4], gj[4];    // where
    // U, S: one sweep, e' = U [e, ghosts] + S r (DD: S acts on the modified rhs, r + C e at the call's start)
    // A: L[e] = A [e, ghosts]
    // M, AM (bottom level): two sweeps of solve_bicgstab2's preconditioner from p * invdiags, and L of that
    const double* m[kTinyMats];
    int off[kTinyMats];  // place in the staged coarse cycle's shared memory (doubles), -1: read from global memory
};
struct CoarseArgs {
    const Lv* lv;        // device array of levels
    int d0;              // level the cycle starts at (vcycle_noinit(d0) semantics)
    int maxdepth;
    int numcycles;
    int nd, nu, nb;      // smoothing counts
    int dd;              // 1: DeferredPoisson2D operators
    const int* refx;     // device arrays, maxdepth entries
    const int* refy;
    int* status;         // device int: 0 ok, nonzero = error code
    const Lv* shadow;    // device array: the levels' layout in shared memory (offsets), or nullptr
    const TinyLv* tiny;  // device array: the levels' dense forms, or nullptr
    int smem_bytes;      // dynamic shared memory the staged levels need
    const double* ainv;  // MGP_FLAG_DIRECT_COARSE: inverse of level maxdepth's operator, transposed, or nullptr
    int grid_ctas;       // > 1: run as a cooperative grid of this many CTAs (gctl set)
    int cluster;         // with grid_ctas > 1: the grid is one thread-block cluster (hardware barriers);
                         // 2: its reductions in the one-CTA kernel's order (the same bits)
    GridCtl gctl;
};

// Largest bottom level solved by its precomputed inverse (cells); b_direct
// gives each row four threads of the coarse CTA.
constexpr int kDirectCells = 64;
// Largest bottom of MGP_FLAG_DIRECT_LARGE (cells): the coarse-cycle level,
// solved by launch_direct_apply.
constexpr int kDirectLargeCells = 1024;
// Pivots per panel of the blocked device Gauss-Jordan (launch_invert); its
// scratch is 4 n^2 + 2 + (n + 1) kGjPanel doubles.
constexpr int kGjPanel = 16;

constexpr int kMaxCoarseLevels = 16;
// Largest staged coarse hierarchy (bytes of dynamic shared memory; the kernels'
// own take 44 KB beside it).
constexpr int kCoarseSmemMax = 180 * 1024;

// Columns of a tiny level's matrices into T.m (device memory), a CTA a column.
// scratch: tiny_scratch_doubles(L) doubles.
size_t tiny_scratch_doubles(const Lv& L);
cudaError_t launch_tiny_columns(const Lv& L, const TinyLv& T, int dd, double* scratch, cudaStream_t st);

// Parameters of the single-CTA BiCGStab (solve_bicgstab2).
struct BicgArgs {
    Lv L;
    DF phi, rhs;
    int homog;
    double tol;
    int max_iters, max_restarts, zerophi;
    int dd;
    int* status;
};

constexpr int kCoarseThreads = 512;   // of the one-CTA coarse cycle: the shape of mgp_sweep.cuh's windows
constexpr int kHeldBottomCells = 5 * kCoarseThreads;   // largest bottom it holds in shared memory
constexpr int kReduceThreads = 256;   // of them that accumulate its reductions
constexpr int kPlainCells = 3600;     // largest level whose general phases are faster in a CTA of that many (mgp_kernels.cu)
constexpr int kGridThreads = 256;     // threads per CTA of the cooperative-grid coarse cycle
constexpr int kClusterThreads = 256;   // threads per CTA of the cluster coarse cycle

long long launch_count();
long long thread_launch_count();   // launches the calling thread made (count_launch on it)
void count_launch(int n = 1);

cudaError_t launch_fill(const DF& p, const Geo& g, const BCd& b, int homog, int do_neum, int nx, int ny,
                        cudaStream_t st);
cudaError_t launch_extrapolate(const DF& p, int nx, int ny, int ngx, int ngy, int order, cudaStream_t st);

// ---- FP32 grid levels of the mixed-precision V-cycle --------------------- //
cudaError_t launch_fill(const DF32& p, const Geo32& g, const BCd& b, int homog, int do_neum, int nx, int ny,
                        cudaStream_t st);
cudaError_t launch_apply(const DF32& out, const DF32& phi, const DF32& rhs, const Geo32& g, const BCd& b, int homog,
                         int nx, int ny, int mode, int jscale, cudaStream_t st);
// Prolongation from an FP32 or an FP64 coarse field (arithmetic in the coarse type).
cudaError_t launch_prolong(const DF32& fine, const DF32& crse, int ncx, int ncy, int refx, int refy, int order,
                           cudaStream_t st);
cudaError_t launch_prolong(const DF32& fine, const DF& crse, int ncx, int ncy, int refx, int refy, int order,
                           cudaStream_t st);
cudaError_t launch_set_guess(const DF32& e, const DF32& r, const DF32& invd, int nx, int ny, cudaStream_t st);
// rc = restrict(rhs - L[phi]) onto the coarse cells, and with guess
// ec = rc * invdc: k_apply (mode 1), the cell restriction and k_set_guess in
// one pass, the same bits.  phi's ghosts must be filled.
cudaError_t launch_resid_restrict(const DF& phi, const DF& rhs, const Geo& g, const BCd& b, int homog, int nx, int ny,
                                  const DF& rc, const DF& ec, const DF& invdc, int ncx, int ncy, int refx, int refy,
                                  int guess, cudaStream_t st);
cudaError_t launch_resid_restrict(const DF32& phi, const DF32& rhs, const Geo32& g, const BCd& b, int homog, int nx,
                                  int ny, const DF32& rc, const DF32& ec, const DF32& invdc, int ncx, int ncy, int refx,
                                  int refy, int guess, cudaStream_t st);
cudaError_t launch_resid_restrict(const DF32& phi, const DF32& rhs, const Geo32& g, const BCd& b, int homog, int nx,
                                  int ny, const DF& rc, const DF& ec, const DF& invdc, int ncx, int ncy, int refx,
                                  int refy, int guess, cudaStream_t st);
// The same with the deferred-correction operator.
cudaError_t launch_dd_resid_restrict(const DF& phi, const DF& rhs, const Geo& g, const BCd& b, int nx, int ny,
                                     const DF& rc, const DF& ec, const DF& invdc, int ncx, int ncy, int refx, int refy,
                                     int guess, cudaStream_t st);
cudaError_t launch_dd_resid_restrict(const DF32& phi, const DF32& rhs, const Geo32& g, const BCd& b, int nx, int ny,
                                     const DF32& rc, const DF32& ec, const DF32& invdc, int ncx, int ncy, int refx, int refy,
                                     int guess, cudaStream_t st);
cudaError_t launch_dd_resid_restrict(const DF32& phi, const DF32& rhs, const Geo32& g, const BCd& b, int nx, int ny,
                                     const DF& rc, const DF& ec, const DF& invdc, int ncx, int ncy, int refx, int refy,
                                     int guess, cudaStream_t st);
cudaError_t launch_sub_mean(const DF32& y, const double* out, int nx, int ny, int gx, int gy, cudaStream_t st);
cudaError_t launch_reduce(int kind, const DF32& a, const DF32& b, int nx, int ny, double vol, double* partials,
                          double* out, cudaStream_t st);
// dst = src rounded to dst's type, over i in [-gx, nx+gx), j in [-gy, ny+gy).
cudaError_t launch_convert(const DF32& dst, const DF& src, int nx, int ny, int gx, int gy, cudaStream_t st);
cudaError_t launch_convert(const DF& dst, const DF32& src, int nx, int ny, int gx, int gy, cudaStream_t st);
cudaError_t launch_round_bf16(const DF32& f, int nx, int ny, int g, cudaStream_t st);
// mode: 0 lap, 1 rhs - lap; jscale divides lap by J first.
cudaError_t launch_apply(const DF& out, const DF& phi, const DF& rhs, const Geo& g, const BCd& b, int homog,
                         int nx, int ny, int mode, int jscale, cudaStream_t st);
cudaError_t launch_gs_sweep(const DF& phi, const DF& rhs, const DF& invd, const Geo& g, const BCd& b, int homog,
                            int nx, int ny, double omega, cudaStream_t st);
// Whether the one-launch sweep serves these sides: DIRI, NEUM or PERIODIC.
bool sweep_fusable(const BCd& b);
// ---- lockstep batches -------------------------------------------------- //
// One launch runs the same phase of many problems.  Each launch has a job
// table and pre[0..njobs]: job k owns blocks [pre[k], pre[k + 1]) of a 1-D
// grid of pre[njobs] blocks (a block finds its job by binary search).
// One sweep's tiles of a large level: regions of gx x gy tiles (a balanced
// partition in pairs of cells), numbered from `first`; inner: away from the
// domain's sides.
struct SweepTiles {
    struct Region {
        int x0, x1, y0, y1, gx, gy, first, inner;
        int px, rx, py, ry;   // pairs of cells a tile, and tiles with one more, along x and y
    };
    int n, total;
    Region r[5];
};
// TMA descriptors of the seven fields a large sweep stages; element (i,j) at
// coordinates (i,j).
struct SweepMaps {
    CUtensorMap phi, rhs, invd, xx, xy, yx, yy;
};
// One level's sweep: phi in buf[flip], written to the other buffer; in_place
// (a level that is one tile): phi in buf[0], swept there.  gx x gy tiles of the
// small shape, or the large shape's tiles.
template <class T>
struct alignas(64) SweepJobT {
    SweepMaps m[2];
    DFT<T> buf[2], rhs, invd;
    GeoT<T> g;
    BCd b;
    SweepTiles tiles;
    int nx, ny, gx, gy, in_place;
};
// fill_ghosts of one field.
template <class T>
struct FillJob {
    DFT<T> p;
    GeoT<T> g;
    BCd b;
    int nx, ny, homog, do_neum;
};
// rc = restrict(rhs - L[phi]), ec = rc * invdc (k_resid_restrict); gbx blocks of 32 x 8 fine cells along x.
template <class T, class TC>
struct ResidJob {
    DFT<T> phi, rhs;
    GeoT<T> g;
    BCd b;
    DFT<TC> rc, ec, invdc;
    int nx, ny, ncx, ncy, refx, refy, gbx;
};
// fine += prolong(crse), order 1 (k_prolong); gbx blocks of 32 x 8 coarse cells along x.
template <class TF, class TC>
struct ProlongJob {
    DFT<TF> fine;
    DFT<TC> crse;
    int ncx, ncy, refx, refy, gbx;
};
// Cell-wise work on the valid region plus g ghost layers (k_cell_jobs: y + x,
// x converted to y's type, y - x, x * z).  gbx blocks of 32 x 8 along x.
template <class TD, class TS>
struct CellJob {
    DFT<TD> y;
    DFT<TS> x;
    DFT<TD> z;
    int nx, ny, g, gbx;
};
// r = rhs - L[phi] on level 0 (caller BCs) and the block's sum of r^2 into
// partials[block]; gbx blocks of 32 x 8 along x.
struct NormJob {
    DF phi, rhs, r;
    Geo g;
    BCd b;
    int nx, ny, homog, gbx;
};
// The coarse cycle of one problem (one CTA each; CoarseArgs with its shadow layout).
struct CoarseJob {
    CoarseArgs a;
};
// e = A^-1 r on a problem's exact bottom (MGP_FLAG_DIRECT_LARGE; k_direct_apply's blocks).
struct DirectJob {
    DF e, r;
    const double* ainv;
    int nx, ny;
};

// How one launch sweeps a level: k sweeps over gx x gy tiles of the small
// shape, or one sweep in the large shape (mgp_sweep.cu).
struct SweepPlan {
    int k, gx, gy;
    bool small;
};
// The small shape's tiles for k sweeps a launch (k = 0: none), and the CTAs of it that run at once.
template <class T>
SweepPlan sweep_tiles(int nx, int ny, int k);
int sweep_wave();
template <class T>
SweepTiles sweep_large_tiles(int nx, int ny);
// A level's descriptors with phi in either of its two buffers.  Built when the
// arrays allow it (16-byte aligned bases and pitches), else ok stays false.
struct LevelMaps {
    SweepMaps a, b;
    const void *pa = nullptr, *pb = nullptr, *rhs = nullptr, *invd = nullptr, *xx = nullptr;
    bool ok = false;
};
void sweep_maps_prepare(LevelMaps* m, const DF& ea, const DF& eb, const DF& rhs, const DF& invd, const Geo& g, int nx,
                        int ny);
void sweep_maps_prepare(LevelMaps* m, const DF32& ea, const DF32& eb, const DF32& rhs, const DF32& invd,
                        const Geo32& g, int nx, int ny);
// The next launch's sweeps when `left` are still to do: 1 <= k <= left.  maps:
// the level's, or nullptr (a caller's arrays).
template <class T>
SweepPlan sweep_plan(int nx, int ny, const BCd& b, int left, const LevelMaps* maps);
// p.k sweeps of a level in one launch, reading pin and writing pout (two
// buffers; the same one is fine when the plan is one tile), with ghosts filled
// at the start of each sweep.  The bits of p.k launches of one sweep.
// dependent: launch as a programmatic dependent of the kernel ahead; the faces
// and invd must not be written by that kernel.  maps as for sweep_plan.  status
// (nullable) receives DST_TIMEOUT if a tile's loads never arrived (not expected).
cudaError_t launch_sweep9(const DF& pin, const DF& pout, const DF& rhs, const DF& invd, const Geo& g, const BCd& b,
                          int homog, int nx, int ny, double omega, const SweepPlan& p, int dependent,
                          const LevelMaps* maps, int* status, cudaStream_t st);
cudaError_t launch_sweep9(const DF32& pin, const DF32& pout, const DF32& rhs, const DF32& invd, const Geo32& g,
                          const BCd& b, int homog, int nx, int ny, double omega, const SweepPlan& p, int dependent,
                          const LevelMaps* maps, int* status, cudaStream_t st);
// Lockstep launches: jobs and pre in device memory (pre[njobs] blocks in all).
template <class T>
cudaError_t launch_sweep9_jobs(const SweepJobT<T>* jobs, const int* pre, int njobs, int nblocks, int k, int small,
                               int flip, int* status, cudaStream_t st);
template <class T>
cudaError_t launch_fill_jobs(const FillJob<T>* jobs, const int* pre, int njobs, int nblocks, int phases,
                             cudaStream_t st);
template <class T, class TC>
cudaError_t launch_resid_jobs(const ResidJob<T, TC>* jobs, const int* pre, int njobs, int nblocks, cudaStream_t st);
template <class TF, class TC>
cudaError_t launch_prolong_jobs(const ProlongJob<TF, TC>* jobs, const int* pre, int njobs, int nblocks,
                                cudaStream_t st);
// kind 0: y = y + x; 1: y = x converted; 2: y = y - x; 3: y = x * z
template <class TD, class TS>
cudaError_t launch_cell_jobs(const CellJob<TD, TS>* jobs, const int* pre, int njobs, int nblocks, int kind,
                             cudaStream_t st);
// r = rhs - L[phi], then norms[k] = sqrt(vol_k * sum of job k's r^2) in block order (vol in volk).
cudaError_t launch_norm_jobs(const NormJob* jobs, const int* pre, int njobs, int nblocks, double* partials,
                             const double* volk, double* norms, cudaStream_t st);
cudaError_t launch_coarse_jobs(const CoarseJob* jobs, int njobs, int smem_bytes, const CoarseJob* plain, int nplain,
                               cudaStream_t st);
int direct_apply_blocks(int nx, int ny);
cudaError_t launch_direct_jobs(const DirectJob* jobs, const int* pre, int njobs, int nblocks, cudaStream_t st);
cudaError_t launch_invdiag(const DF& invd, const Geo& g, const BCd& b, int homog, int nx, int ny, int coupled,
                           cudaStream_t st);
// kind: 0 cell, 1 x-face, 2 y-face, 3 node.  ncx/ncy = coarse cell counts.
cudaError_t launch_restrict(const DF& f, const DF& c, int ncx, int ncy, int refx, int refy, int kind,
                            cudaStream_t st);
// Constant, linear and (order 2) second-difference terms; crse ghosts must be filled.
cudaError_t launch_prolong(const DF& fine, const DF& crse, int ncx, int ncy, int refx, int refy, int order,
                           cudaStream_t st);
cudaError_t launch_prolong_cross(const DF& fine, const DF& crse, int ncx, int ncy, cudaStream_t st);
cudaError_t launch_set_guess(const DF& e, const DF& r, const DF& invd, int nx, int ny, cudaStream_t st);
cudaError_t launch_jacobi(const DF& phi, const DF& r, const DF& invd, double omega, int nx, int ny, cudaStream_t st);
// y[i,j] = a*y + b*x over i in [-gx, nx+gx), j in [-gy, ny+gy).
// A set of vectors for GMRES: vector k at p + k * stride, cell (i,j) at [i + j * ld].
struct MVec {
    double* p;
    int ld;
    long stride;
};
// out[k] = sum over valid cells of w * v_k, k < nv (partials: nb * nv doubles).
cudaError_t launch_mdot(const DF& w, const MVec& V, int nv, int nx, int ny, double* partials, int nb, double* out,
                        cudaStream_t st);
// One classical Gram-Schmidt pass: h[k] = w . v_k (k < nv), w -= sum_k h[k] v_k,
// then *hnorm = |w|^2.  partials holds cap doubles; cudaErrorNotSupported
// when the pass's partial sums would not fit (the caller then uses
// launch_mdot and launch_maxpy).
cudaError_t launch_gs_pass(const DF& w, const MVec& V, int nv, int nx, int ny, double* partials, long cap, int nb,
                           double* h, double* hnorm, cudaStream_t st);
// w += sign * sum_{k < nv} coef[k] v_k (coef in device memory).
cudaError_t launch_maxpy(const DF& w, const MVec& V, int nv, const double* coef, double sign, int nx, int ny,
                         cudaStream_t st);
cudaError_t launch_axpby(const DF& y, const DF& x, double a, double b, int nx, int ny, int gx, int gy,
                         cudaStream_t st);
// y = y * x (mul=1) or y / x (mul=0) over the valid region.
cudaError_t launch_muldiv(const DF& y, const DF& x, int mul, int nx, int ny, cudaStream_t st);
cudaError_t launch_fillval(const DF& y, double v, int nx, int ny, int gx, int gy, cudaStream_t st);
cudaError_t launch_sub_mean(const DF& y, const double* out, int nx, int ny, int gx, int gy, cudaStream_t st);
// Reduction over the valid region into out[0] (and out[1] for RED_JSUM: volume).
cudaError_t launch_reduce(int kind, const DF& a, const DF& b, int nx, int ny, double vol, double* partials,
                          double* out, cudaStream_t st);
// Gradient and divergence (compute_pd, compute_grad, compute_div,
// fill_boundary_fluxes); phi's ghosts filled by the caller.
cudaError_t launch_pd(const DF& pd, const DF& phi, int nx, int ny, double dx, double dy, int dir, int nodedir,
                      cudaStream_t st);
cudaError_t launch_grad(const DF& xflux, const DF& yflux, const DF& phi, const Geo& g, const BCd& b, int homog,
                        int nx, int ny, cudaStream_t st);
cudaError_t launch_boundary_fluxes(const DF& xflux, const DF& yflux, const BCd& b, int homog, int nx, int ny,
                                   cudaStream_t st);
cudaError_t launch_div(const DF& div, const DF& xflux, const DF& yflux, int nx, int ny, double dx, double dy,
                       cudaStream_t st);
// Deferred-correction operators.
cudaError_t launch_dd_invdiag(const DF& invd, const Geo& g, int nx, int ny, cudaStream_t st);
cudaError_t launch_dd_modrhs(const DF& out, const DF& phi, const DF& rhs, const Geo& g, int nx, int ny,
                             cudaStream_t st);
cudaError_t launch_dd_colour(const DF& phi, const DF& modrhs, const DF& invd, const Geo& g, int nx, int ny,
                             double omega, int colour, cudaStream_t st);
// Several red-black sweeps (ghost fill included) in one launch, pin to pout (two
// buffers) for the modified rhs m; *done of the `left` sweeps were launched.  A
// programmatic dependent: the faces and invd must not be written by the kernel
// ahead.  Sides must be Dirichlet or Neumann with LAH ghosts (dd_sweep_fusable);
// the solver's own arrays (rows aligned to pairs).
bool dd_sweep_fusable(const BCd& b);
cudaError_t launch_dd_sweeps(const DF& pin, const DF& pout, const DF& m, const DF& invd, const Geo& g, const BCd& b,
                             int nx, int ny, double omega, int left, int* done, cudaStream_t st);
cudaError_t launch_dd_sweeps(const DF32& pin, const DF32& pout, const DF32& m, const DF32& invd, const Geo32& g,
                             const BCd& b, int nx, int ny, double omega, int left, int* done, cudaStream_t st);
// modrhs and colour on FP32 fields (the grid levels of a mixed-precision DD V-cycle).
cudaError_t launch_dd_modrhs(const DF32& out, const DF32& phi, const DF32& rhs, const Geo32& g, int nx, int ny,
                             cudaStream_t st);
cudaError_t launch_dd_colour(const DF32& phi, const DF32& modrhs, const DF32& invd, const Geo32& g, int nx, int ny,
                             double omega, int colour, cudaStream_t st);
// Per-device kernel attributes (idempotent; call before any stream capture).
cudaError_t sweep_kernels_init();
cudaError_t coarse_kernels_init();
// Single-CTA kernels.
cudaError_t launch_coarse_cycle(const CoarseArgs& a, cudaStream_t st);
// Largest cooperative grid of the coarse cycle the current device keeps resident (0: none).
int coarse_grid_ctas_max();
int coarse_cluster_ctas_max();
// A cooperative grid of nctas CTAs (all resident) passing nbar grid barriers;
// CTA `skip` (if >= 0) exits before the first one, so the others' waits run
// out.  Exercises the bounded wait of the coarse cycle's grid barrier.
cudaError_t launch_barrier_selftest(const GridCtl& g, int nctas, int skip, int nbar, cudaStream_t st);
int barrier_selftest_ctas_max();
// A[m * n + k] = (L e_k)_m for the level's operator with homogeneous BCs
// (n = nx * ny columns, one CTA each; scratch holds 2 n fields of
// (nx + 2) x (ny + 2)).
cudaError_t launch_direct_columns(const Lv& L, double* scratch, double* A, cudaStream_t st);
// Inverse of the n x n row-major A by Gauss-Jordan elimination with partial
// pivoting on the device, into ainv (row-major, may alias A).  work holds
// 4 n^2 + 2 + (n + 1) kGjPanel doubles (16-byte aligned), iwork 2 n + 1 ints;
// *fail (in iwork) ends nonzero when a pivot fell below 1e-13 of the largest
// |A| entry (singular to working precision).  Launches 2 n / kGjPanel + 2
// kernels.
cudaError_t launch_invert(const double* A, int n, double* ainv, double* work, int* iwork, cudaStream_t st);
// e = ainv r on the level's cells (n = nx * ny <= kDirectLargeCells; cells
// numbered i fastest), one warp per row.
cudaError_t launch_direct_apply(const DF& e, const DF& r, const double* ainv, int nx, int ny, cudaStream_t st);
cudaError_t launch_bicgstab(const BicgArgs& a, cudaStream_t st);

// The exact bottom of a level of more than kDirectLargeCells cells (mgp_bottom.cu):
// block cyclic reduction over its lines of m cells.
constexpr int kBlockLineMax = 160;                  // an inverted block fits one CTA's shared memory
constexpr int kBlockLinesMax = 16384;
constexpr int kBlockStepsMax = 16;
constexpr size_t kBlockBytesMax = 256ull << 20;     // of factors
struct BlockBottom {
    int m, lines, along_y, steps;                   // lines are rows (along_y) or columns of the level
    int ndown[kBlockStepsMax + 1], odown[kBlockStepsMax + 1], nup[kBlockStepsMax + 1], oup[kBlockStepsMax + 1];
    double *mem, *dinv, *p, *q, *fg, *r;            // one block of memory, nullptr without a factorisation
    int4* items;
    size_t bytes;
};
struct BlockAlloc {
    void* (*get)(void* ctx, size_t bytes);          // nullptr when there is no memory
    void (*put)(void* ctx, void* p);
    void* ctx;
};
// Whether a level of these sides and types has such a bottom; sets its shape.
bool block_bottom_shape(int nx, int ny, const BCd& bc, BlockBottom* b);
// Device bytes its set-up needs at its most (the factors and the scratch beside them); 0 without such a bottom.
size_t block_bottom_peak_bytes(int nx, int ny, const BCd& bc);
// Factorises the level's operator (homogeneous sides) and tries it; synchronises st.
// *ok: it solves.  Without memory or a sound factorisation *b is empty.
cudaError_t block_bottom_build(BlockBottom* b, const Geo& g, const BCd& bc, int nx, int ny, const BlockAlloc& mem,
                               cudaStream_t st, bool* ok);
// e = A^-1 r on the level's cells (ghosts untouched).
cudaError_t launch_block_bottom(const BlockBottom& b, const DF& e, const DF& r, cudaStream_t st);
// The same for many levels at once (lockstep batches): the launches of the longest
// reduction, each a step of every problem that has it, steps 0 .. down and then
// .. 0 up, in the same bits.  Blocks of a problem in a step, and the step's launch.
struct BlockJob {
    BlockBottom b;
    DF e, r;
};
int block_bottom_blocks(const BlockBottom& b, int l, bool up);
cudaError_t launch_block_jobs(const BlockJob* jobs, const int* pre, int njobs, int nblocks, int l, bool up,
                              cudaStream_t st);

}  // namespace mgp
