// mgp_sweep.cu -- Gauss-Seidel sweeps of the mapped 9-point operator, one or
// several per launch (relax_gs, poisson2d.f90:1460-1988, in the device order).
//
// A launch reads phi from `pin` and writes the swept field to `pout` (two
// buffers), so no CTA reads a value another CTA has already replaced; a level
// that one CTA covers may be swept in place.  A CTA owns a tile of a balanced
// partition of the grid and works on a window of cells around it.  A sweep's
// sub-passes are
//   * the sweep-start ghost fill (P2:1556);
//   * the four colours (0,0),(1,1),(1,0),(0,1) over interior cells;
//   * along the domain's non-periodic sides the edge cells colour by colour,
//     then the four corners.
// Every pass runs on the whole window: what it computes near the window's rim
// from cells the window does not hold is wrong, and moves inward by a known
// number of cells a pass, never into the tile.  With K sweeps a window has 4 K +
// 2 columns left of its tile, 4 K right and 4 K + 2 rows below and above (tiles
// start at even cells; tests/test_sweep_halo.py walks the dependences of every
// partition shape).  So K sweeps in a launch give the bits of K launches, and
// the result depends on neither the tiling nor K.
//
// The operator lives in registers.  A thread owns a 2 x 2 block of cells -- one
// of each colour -- and keeps their face coefficients, inverse diagonals and
// right-hand sides (32 values, 36 with phi) through all K sweeps.  Shared memory holds
// phi alone, as four planes, one per colour (i mod 2, j mod 2), so a colour pass
// reads its five neighbours outside the block with consecutive lanes on
// consecutive words.  (With the whole operator in shared memory at one word a
// cell, a colour reads 19 values an update at stride two: 640 of the ~900
// cycles of a pass with one CTA on the SM were replayed wavefronts, and the
// edge cells, one generic routine for four sides, another 0.5 us a colour.)
//
// Two shapes, chosen by sweep_plan.  Levels whose sweeps last one CTA's latency
// take several sweeps a launch, with four warps of their own for the sides:
// measured per sweep of an n^2 level, FP32 / FP64, before (operator in shared
// memory, two sweeps a launch) and now: 128^2 8.4 / 8.3 -> 2.2 / 3.4 us, 256^2
// 8.5 / 8.3 -> 2.3 / 5.2 us, 512^2 8.7 / 11 -> 5.7 / 9.9 us.  Large levels take
// one sweep a launch by persistent CTAs that load the next tile while they
// sweep one: 1024^2 17.2 / 32 -> 13 / 22 us, 2048^2 41 / 88 -> 37 / 72 us
// (0.57 / 0.58 of the copy rate by the 8 words a cell of a sweep).  They are
// bound by the barriers between colour passes (5 of 18 cycles between a warp's
// issues), not by the bytes; the small ones by the sides (mgp_sweep.cuh).
#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <mutex>
#include <type_traits>

#include "mgp_kernels.cuh"
#include "mgp_stage.cuh"
#include "mgp_sweep.cuh"

namespace mgp {

namespace {

// K sweeps of a tile by a CTA of its own.
template <class C, bool kVec, class T>
__device__ __forceinline__ void sweep_tile(const DFT<T>& pin, const DFT<T>& pout, const DFT<T>& rhs,
                                           const DFT<T>& invd, const GeoT<T>& g, const BCd& b, int homog, int nx,
                                           int ny, int gx, int gy, double omega, int K, int bx, int by) {
    __shared__ T s[4 * C::PS];
    __shared__ T strips[4 * kStrip * kAlong];
    sweep_window<C, kVec, false>(s, strips, pin, pout, rhs, invd, g, b, homog, nx, ny, gx, gy, omega, K, bx, by);
}

// ---- one sweep of a large level -------------------------------------------- //
// A persistent CTA walks over tiles and, while it sweeps one, has the next
// one's operands on the way: a thread issues seven TMA tile loads (the window
// of phi, rhs, the inverse diagonal and the four faces) into one staging buffer
// that is free again as soon as the threads have taken their blocks into
// registers, so the loads' latency is off the chain of colour passes and their
// addresses off the instruction stream (with a cp.async a row and array instead,
// 690 instructions a thread and tile and 57.7 us at 2048^2 in FP32).
template <class C>
struct Stage {
    using T = typename C::T;
    static constexpr int kAlign = 16 / (int)sizeof(T);                // a TMA load starts at a multiple of 16 bytes
    static constexpr int PW = (C::WX + 1 + (kAlign - 2) + kAlign - 1) / kAlign * kAlign;   // the window and a face
    static constexpr int PH = C::WY + 1;
    static constexpr int kA = (PW * PH * (int)sizeof(T) + 127) / 128 * 128 / (int)sizeof(T);   // 128-byte aligned
    static constexpr unsigned kBytes = PW * PH * sizeof(T);
    enum { A_XX, A_XY, A_YX, A_YY, A_D, A_P, A_F, kArrays };
    static constexpr size_t kSmem = (size_t)kArrays * kA * sizeof(T) + 128;
};

// A CTA gives up on its tile loads after kWaitLimit polls or kWaitNs, far
// above any real wait (microseconds); a poll sleeps up to kSuspendNs.
constexpr long kWaitLimit = 1L << 22;
constexpr unsigned long long kWaitNs = 200000000ull;
constexpr unsigned kSuspendNs = 20000;

__device__ __forceinline__ void mbar_init(unsigned bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(unsigned bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity), "r"(kSuspendNs)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// Bounded wait for the barrier's phase of the given parity; false if it did not complete.
__device__ __forceinline__ bool mbar_wait(unsigned bar, unsigned parity) {
    if (mbar_try_wait(bar, parity)) return true;
    const unsigned long long t0 = global_ns();
    for (long k = 0; k < kWaitLimit; ++k) {
        if (mbar_try_wait(bar, parity)) return true;
        if (global_ns() - t0 > kWaitNs) break;
    }
    return false;
}
// One 2-D tile (the map's box) of `map` at element coordinates (x, y); x is a
// multiple of 16 bytes.
__device__ __forceinline__ void tma_load_2d(unsigned dst, const CUtensorMap* map, int x, int y, unsigned bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n"
        ::"r"(dst), "l"((unsigned long long)map), "r"(x), "r"(y), "r"(bar)
        : "memory");
}

// The next tile, as the thread that places it leaves it for the others.
struct NextTile {
    int t, job, inner;   // t < 0: none
    Window w;
};

// Tile t of a level's partition; true for a tile of the inner region, whose
// whole window lies inside the domain, off its sides.
__device__ __forceinline__ bool place_tile(const SweepTiles& S, int t, int nx, int ny, Window& w) {
    int r = 0;
    while (r + 1 < S.n && t >= S.r[r + 1].first) ++r;
    const SweepTiles::Region& R = S.r[r];
    const int q = t - R.first, by = q / R.gx, bx = q - by * R.gx;
    const int X0 = R.x0 + 2 * (bx * R.px + min(bx, R.rx)), X1 = min(R.x1, X0 + 2 * (R.px + (bx < R.rx)));
    const int Y0 = R.y0 + 2 * (by * R.py + min(by, R.ry)), Y1 = min(R.y1, Y0 + 2 * (R.py + (by < R.ry)));
    if (R.inner) w.set(X0, X1, Y0, Y1, 4, 2, 4, 4, nx, ny);
    else w.set(X0, X1, Y0, Y1, 6, 4, 6, 6, nx, ny);
    return R.inner;
}

// A level as a large sweep's CTA sees it.
template <class T>
struct LevelRef {
    const DFT<T>*pin, *pout;
    const GeoT<T>* g;
    const BCd* b;
    int nx, ny;
};

// One sweep of the tiles blockIdx.x, blockIdx.x + gridDim.x, ... below total.
// find(t, job, inner, window) places tile t (job: in, the level of the tile
// before); level(job) gives its level, maps(job) its descriptors.
template <class C, class T, class Find, class Level, class Maps>
__device__ __forceinline__ void sweep_stream(int total, int homog, double omega, int* status, Find find, Level level,
                                             Maps maps) {
    using S = Stage<C>;
    using V = typename Pair<T>::type;
    __shared__ T s[4 * C::PS];
    __shared__ T strips[4 * kStrip * kAlong];
    __shared__ NextTile tiles[2];
    __shared__ LevelRef<T> levels[2];
    __shared__ int bad;
    __shared__ __align__(8) unsigned long long barrier_word;
    extern __shared__ unsigned char stage_raw[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int kbx = tid % C::LB, kby = tid / C::LB;
    T* stage = reinterpret_cast<T*>(stage_raw + ((128 - ((unsigned)__cvta_generic_to_shared(stage_raw) & 127)) & 127));
    const unsigned sb = (unsigned)__cvta_generic_to_shared(stage), bar = (unsigned)__cvta_generic_to_shared(&barrier_word);
    T* own = s + (kby + 1) * C::P + kbx + 1;
    const bool issuer = tid == C::kThreads - 32;   // the last warp serves no side
    const auto load_const = [&](const NextTile& n) {
        const SweepMaps& m = *maps(n.job);
        const int x = n.w.ox & ~(S::kAlign - 1);
        mbar_expect_tx(bar, S::kArrays * S::kBytes);
        tma_load_2d(sb + S::A_XX * S::kA * sizeof(T), &m.xx, x, n.w.oy, bar);
        tma_load_2d(sb + S::A_XY * S::kA * sizeof(T), &m.xy, x, n.w.oy, bar);
        tma_load_2d(sb + S::A_YX * S::kA * sizeof(T), &m.yx, x, n.w.oy, bar);
        tma_load_2d(sb + S::A_YY * S::kA * sizeof(T), &m.yy, x, n.w.oy, bar);
        tma_load_2d(sb + S::A_D * S::kA * sizeof(T), &m.invd, x, n.w.oy, bar);
    };
    const auto load_fields = [&](const NextTile& n) {
        const SweepMaps& m = *maps(n.job);
        const int x = n.w.ox & ~(S::kAlign - 1);
        tma_load_2d(sb + S::A_P * S::kA * sizeof(T), &m.phi, x, n.w.oy, bar);
        tma_load_2d(sb + S::A_F * S::kA * sizeof(T), &m.rhs, x, n.w.oy, bar);
    };
    if (issuer) {
        mbar_init(bar, 1);
        bad = 0;
        NextTile& n = tiles[0];
        n.t = blockIdx.x;
        n.job = 0;
        find(n);
        levels[0] = level(n.job);
        load_const(n);   // constant during a solve: requested before the wait for the kernel ahead
    }
    grid_dependency_wait();
    if (issuer) load_fields(tiles[0]);
    cta_sync();
    // One tile; kInner: of the inner region, without sides.  (Two copies: the
    // sides' code takes so many registers that the FP32 kernel spills, which the
    // inner tiles then do not see.)
    const auto tile = [&](auto inner_tag, int it) -> TileEnd {
        constexpr bool kInner = decltype(inner_tag)::value;
        const Window& w = tiles[it].w;
        const LevelRef<T>& L0 = levels[it];
        const T idx = T(L0.g->idx), idy = T(L0.g->idy), om = T(omega), om1 = T(1.0 - omega);
        Block<T> k;
        {
            const T* q = stage + 2 * kby * S::PW + (w.ox & (S::kAlign - 1)) + 2 * kbx;
#pragma unroll
            for (int r = 0; r < 3; ++r) {
                const auto get = [&](int a, T& v0, T& v1) {
                    const V v = *reinterpret_cast<const V*>(q + a * S::kA + r * S::PW);
                    v0 = v.x;
                    v1 = v.y;
                };
                get(S::A_YX, k.yx[r][0], k.yx[r][1]);
                get(S::A_YY, k.yy[r][0], k.yy[r][1]);
                if (r < 2) {
                    get(S::A_XX, k.xx[r][0], k.xx[r][1]);
                    get(S::A_XY, k.xy[r][0], k.xy[r][1]);
                    get(S::A_D, k.d[r][0], k.d[r][1]);
                    get(S::A_P, k.p[r][0], k.p[r][1]);
                    get(S::A_F, k.f[r][0], k.f[r][1]);
                    k.xx[r][2] = q[S::A_XX * S::kA + r * S::PW + 2];
                    k.xy[r][2] = q[S::A_XY * S::kA + r * S::PW + 2];
                }
            }
        }
        const bool any_side = !kInner && w.any();
        if (any_side) fixed_ghosts<C>(s, w, *L0.pin, *L0.b, L0.nx, L0.ny);
        const unsigned mask =
            settle<C, kInner>(k, s, strips, w, kbx, kby, idx, idy, om, *L0.b, L0.nx, L0.ny);
        cta_sync();   // the planes are in place, the staging buffer is read and the next tile placed
        // A thread gave up on the loads, so what was read may be anything: nothing is
        // stored.  (Decided at this barrier, which the tile needs anyway, not at one
        // of its own before the staging buffer is read.)
        if (bad) return TILE_LOST;
        const bool more = tiles[it ^ 1].t >= 0;
        if (issuer && more) {
            load_const(tiles[it ^ 1]);
            load_fields(tiles[it ^ 1]);
        }
        if (any_side) {
            if (plain_sides(*L0.b, homog)) {
                with_side<C>(warp, w, L0.nx, L0.ny, [&](auto L) {
                    L.place(w, *L0.g, *L0.b, homog, L0.nx, L0.ny, om, om1);
                    L.grab(s);
                    L.put(s);
                });
                cta_sync();
            }
            reload<C>(k, own);
        }
        colours<C>(k, own, mask, idx, idy, om, om1);
        if (any_side) {
            with_side<C>(warp, w, L0.nx, L0.ny, [&](auto L) {
                L.place(w, *L0.g, *L0.b, homog, L0.nx, L0.ny, om, om1);
                L.take(strips, w, *L0.b, homog);
                L.pass(s, strips, w, *L0.g, *L0.b, homog, L0.nx, L0.ny);
            });
            cta_sync();
            reload<C>(k, own);
            store_ghosts<C>(s, *L0.pout, w, warp, L0.nx, L0.ny);
        }
        store_block<true>(k, *L0.pout, w, w.ox + 2 * kbx, w.oy + 2 * kby);
        if (more) cta_sync();   // the planes are read no more
        return more ? TILE_MORE : TILE_LAST;
    };
    walk_tiles(
        [&](int it) {   // while this tile's loads are in flight: ghosts they do not make, and the next tile
            const LevelRef<T>& L0 = levels[it];
            if (warp < 4 && !tiles[it].inner)
                start_ghosts<C>(s, tiles[it].w, *L0.pin, *L0.b, homog, L0.nx, L0.ny, warp);
            if (!issuer) return;
            NextTile& n = tiles[it ^ 1];
            n.t = tiles[it].t + gridDim.x;
            n.job = tiles[it].job;
            if (n.t < total) {
                find(n);
                levels[it ^ 1] = level(n.job);
            } else {
                n.t = -1;
            }
        },
        [&](unsigned parity) {
            if (mbar_wait(bar, parity)) return;
            bad = 1;   // never seen
            if (lane == 0) set_status(status, DST_TIMEOUT);
        },
        [&](int it) { return tiles[it].inner ? tile(std::true_type(), it) : tile(std::false_type(), it); },
        [&](unsigned parity) {   // let copies still in flight land before the CTA exits
            if (issuer) mbar_wait(bar, parity);
        });
}

template <class C>
__global__ void __launch_bounds__(C::kThreads, C::kMinBlocks)
    k_sweep9_stream(const __grid_constant__ SweepMaps m, const __grid_constant__ DFT<typename C::T> pin,
                    const __grid_constant__ DFT<typename C::T> pout, const __grid_constant__ GeoT<typename C::T> g,
                    const __grid_constant__ BCd b, const __grid_constant__ SweepTiles tiles, int homog, int nx, int ny,
                    double omega, int* status) {
    using T = typename C::T;
    allow_dependents();
    const SweepMaps* const mp = &m;
    sweep_stream<C, T>(
        tiles.total, homog, omega, status, [&](NextTile& n) { n.inner = place_tile(tiles, n.t, nx, ny, n.w); },
        [&](int) { return LevelRef<T>{&pin, &pout, &g, &b, nx, ny}; }, [mp](int) { return mp; });
}

// The same over the levels of many problems (lockstep batches).  Descriptors in
// a job table may have been rewritten since the last launch that read them
// (tables are rebuilt when the set of unconverged problems changes): the
// tensor-map proxy is made to see the new ones before use.
template <class C>
__global__ void __launch_bounds__(C::kThreads, C::kMinBlocks)
    k_sweep9_stream_jobs(const SweepJobT<typename C::T>* __restrict__ jobs, const int* __restrict__ pre, int njobs,
                         int total, int flip, int* status) {
    using T = typename C::T;
    allow_dependents();
    sweep_stream<C, T>(
        total, 1, 1.0, status,
        [&](NextTile& n) {
            const bool first = n.t < (int)gridDim.x;
            int job = n.job;
            while (job + 1 < njobs && __ldg(pre + job + 1) <= n.t) ++job;   // a CTA's tiles come in order
            if (first || job != n.job) {
                const SweepMaps& m = jobs[job].m[flip];
                for (const CUtensorMap* d : {&m.phi, &m.rhs, &m.invd, &m.xx, &m.xy, &m.yx, &m.yy})
                    asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(d) : "memory");
            }
            n.job = job;
            const SweepJobT<T>& J = jobs[job];
            n.inner = place_tile(J.tiles, n.t - __ldg(pre + job), J.nx, J.ny, n.w);
        },
        [&](int job) {
            const SweepJobT<T>& J = jobs[job];
            return LevelRef<T>{&J.buf[flip], &J.buf[flip ^ 1], &J.g, &J.b, J.nx, J.ny};
        },
        [&](int job) { return &jobs[job].m[flip]; });
}

template <class C, bool kVec>
__global__ void __launch_bounds__(C::kThreads, C::kMinBlocks)
    k_sweep9(DFT<typename C::T> pin, DFT<typename C::T> pout, DFT<typename C::T> rhs, DFT<typename C::T> invd,
             GeoT<typename C::T> g, const __grid_constant__ BCd b, int homog, int nx, int ny, double omega, int K) {
    allow_dependents();
    sweep_tile<C, kVec>(pin, pout, rhs, invd, g, b, homog, nx, ny, gridDim.x, gridDim.y, omega, K, blockIdx.x,
                        blockIdx.y);
}

// Lockstep batches: one launch sweeps the same level of many problems.  Job
// k owns blocks [pre[k], pre[k + 1]) of the grid, one per tile of its level
// (row-major over its gx x gy tiles); a block finds its job by binary
// search.  flip selects the buffer each job's phi is read from, so one job
// table serves every sweep of a smoothing call; a job whose level is one tile
// is swept in place.
template <class C>
__global__ void __launch_bounds__(C::kThreads, C::kMinBlocks)
    k_sweep9_jobs(const SweepJobT<typename C::T>* __restrict__ jobs, const int* __restrict__ pre, int njobs, int K,
                  int flip) {
    allow_dependents();
    const int blk = blockIdx.x;
    int lo = 0, hi = njobs - 1;
    while (lo < hi) {   // the last job with pre[job] <= blk
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(pre + mid) <= blk) lo = mid;
        else hi = mid - 1;
    }
    const SweepJobT<typename C::T>& J = jobs[lo];
    const int q = blk - __ldg(pre + lo), side = J.in_place ? 0 : flip;
    sweep_tile<C, true>(J.buf[side], J.buf[J.in_place ? 0 : side ^ 1], J.rhs, J.invd, J.g, J.b, 1, J.nx, J.ny, J.gx,
                        J.gy, 1.0, K, q % J.gx, q / J.gx);
}

int sm_count() {
    static std::mutex mu;
    static int n[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
    std::lock_guard<std::mutex> lock(mu);
    if (!n[dev] && cudaDeviceGetAttribute(&n[dev], cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
        cudaGetLastError();
        n[dev] = 148;
    }
    return n[dev];
}

template <class T>
bool pair_aligned(const DFT<T>& f) {
    return (reinterpret_cast<uintptr_t>(f.p) & (2 * sizeof(T) - 1)) == 0 && (f.ld & 1) == 0;
}

// The shapes in use: several sweeps a launch of small levels, and one sweep a
// launch of large ones.
using Small32 = Shape<float, 28, 32, true, 1>;
using Large32 = Shape<float, 16, 32, false, 2>;
using Large64 = Shape<double, 16, 32, false, 1>;
template <class T>
struct Shapes;
template <>
struct Shapes<float> {
    using Small = Small32;
    using Large = Large32;
};
template <>
struct Shapes<double> {
    using Small = Small64;
    using Large = Large64;
};

cudaLaunchConfig_t config(dim3 grid, int threads, size_t smem, int dependent, cudaLaunchAttribute* at,
                          cudaStream_t st) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    at->id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at->val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = dependent ? 1 : 0;
    return cfg;
}

template <class T>
const SweepMaps* maps_for(const LevelMaps* m, const DFT<T>& pin, const DFT<T>& rhs, const DFT<T>& invd,
                          const GeoT<T>& g) {
    if (!m || !m->ok || (const void*)rhs.p != m->rhs || (const void*)invd.p != m->invd || (const void*)g.xx.p != m->xx)
        return nullptr;
    return (const void*)pin.p == m->pa ? &m->a : (const void*)pin.p == m->pb ? &m->b : nullptr;
}

template <bool kVec, class T>
cudaError_t launch_any(const DFT<T>& pin, const DFT<T>& pout, const DFT<T>& rhs, const DFT<T>& invd,
                       const GeoT<T>& g, const BCd& b, int homog, int nx, int ny, double omega, const SweepPlan& p,
                       int dependent, const LevelMaps* maps, int* status, cudaStream_t st) {
    using S = typename Shapes<T>::Small;
    using L = typename Shapes<T>::Large;
    cudaLaunchAttribute at;
    if (p.small) {
        const cudaLaunchConfig_t cfg = config(dim3(p.gx, p.gy), S::kThreads, 0, dependent, &at, st);
        return cudaLaunchKernelEx(&cfg, k_sweep9<S, kVec>, pin, pout, rhs, invd, g, b, homog, nx, ny, omega, p.k);
    }
    const SweepMaps* m = maps_for(maps, pin, rhs, invd, g);
    if (!m) return cudaErrorInvalidValue;
    const SweepTiles tiles = sweep_large_tiles<T>(nx, ny);
    const int ctas = std::min(tiles.total, L::kMinBlocks * sm_count());
    const cudaLaunchConfig_t cfg = config(dim3(ctas), L::kThreads, Stage<L>::kSmem, dependent, &at, st);
    return cudaLaunchKernelEx(&cfg, k_sweep9_stream<L>, *m, pin, pout, g, b, tiles, homog, nx, ny, omega, status);
}

template <class T>
cudaError_t sweep_impl(const DFT<T>& pin, const DFT<T>& pout, const DFT<T>& rhs, const DFT<T>& invd,
                       const GeoT<T>& g, const BCd& b, int homog, int nx, int ny, double omega, const SweepPlan& p,
                       int dependent, const LevelMaps* maps, int* status, cudaStream_t st) {
    const DFT<T> fields[] = {pin, pout, rhs, invd, g.xx, g.xy, g.yx, g.yy};
    bool vec = true;
    for (const DFT<T>& f : fields) vec = vec && pair_aligned(f);
    cudaError_t e = sweep_kernels_init();
    if (e != cudaSuccess) return e;
    if (vec) e = launch_any<true>(pin, pout, rhs, invd, g, b, homog, nx, ny, omega, p, dependent, maps, status, st);
    else if constexpr (sizeof(T) == 8) e = launch_any<false>(pin, pout, rhs, invd, g, b, homog, nx, ny, omega, p, dependent, maps, status, st);
    else e = cudaErrorMisalignedAddress;   // FP32 fields are the solver's own, always aligned
    count_launch();
    return e;
}

template <class C>
SweepPlan tiles_of(int nx, int ny, int k) {
    SweepPlan p;
    p.k = k;
    p.small = true;
    // a direction the window covers whole needs no halo
    p.gx = nx <= C::WX ? 1 : ((nx + 1) / 2 + C::tx(k) / 2 - 1) / (C::tx(k) / 2);
    p.gy = ny <= C::WY ? 1 : ((ny + 1) / 2 + C::ty(k) / 2 - 1) / (C::ty(k) / 2);
    return p;
}

template <class F>
cudaError_t allow_smem(F* k, size_t bytes) {
    return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

}  // namespace

// Per device: dynamic shared memory above 48 KB must be opted into (before any
// stream capture).
cudaError_t sweep_kernels_init() {
    static std::mutex mu;
    static unsigned long long done = 0;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lock(mu);
    if (dev < 64 && (done >> dev) & 1ull) return cudaSuccess;
    e = allow_smem(k_sweep9_stream<Large32>, Stage<Large32>::kSmem);
    if (e == cudaSuccess) e = allow_smem(k_sweep9_stream_jobs<Large32>, Stage<Large32>::kSmem);
    if (e == cudaSuccess) e = allow_smem(k_sweep9_stream<Large64>, Stage<Large64>::kSmem);
    if (e == cudaSuccess) e = allow_smem(k_sweep9_stream_jobs<Large64>, Stage<Large64>::kSmem);
    if (e == cudaSuccess && dev < 64) done |= 1ull << dev;
    return e;
}

namespace {

PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
        else
            cudaGetLastError();
    });
    return fn;
}

// A 2-D map of the width x height elements of f, box the large shape's window.
template <class T>
bool encode(CUtensorMap* m, const DFT<T>& f, int width, int height) {
    using S = Stage<typename Shapes<T>::Large>;
    const PFN_cuTensorMapEncodeTiled_v12000 fn = encode_fn();
    if (!fn || ((uintptr_t)f.p & 15) || (((long)f.ld * (long)sizeof(T)) & 15)) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)width, (cuuint64_t)height};
    const cuuint64_t strides[1] = {(cuuint64_t)f.ld * sizeof(T)};
    const cuuint32_t box[2] = {(cuuint32_t)S::PW, (cuuint32_t)S::PH};
    const cuuint32_t es[2] = {1, 1};
    return fn(m, sizeof(T) == 8 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT64 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, f.p, dims,
              strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <class T>
void prepare(LevelMaps* m, const DFT<T>& ea, const DFT<T>& eb, const DFT<T>& rhs, const DFT<T>& invd,
             const GeoT<T>& g, int nx, int ny) {
    m->ok = encode(&m->a.phi, ea, nx, ny) && encode(&m->b.phi, eb, nx, ny) && encode(&m->a.rhs, rhs, nx, ny) &&
            encode(&m->a.invd, invd, nx, ny) && encode(&m->a.xx, g.xx, nx + 1, ny) &&
            encode(&m->a.xy, g.xy, nx + 1, ny) && encode(&m->a.yx, g.yx, nx, ny + 1) &&
            encode(&m->a.yy, g.yy, nx, ny + 1);
    const CUtensorMap phi = m->b.phi;
    m->b = m->a;
    m->b.phi = phi;
    m->pa = ea.p;
    m->pb = eb.p;
    m->rhs = rhs.p;
    m->invd = invd.p;
    m->xx = g.xx.p;
}

}  // namespace

void sweep_maps_prepare(LevelMaps* m, const DF& ea, const DF& eb, const DF& rhs, const DF& invd, const Geo& g, int nx,
                        int ny) {
    prepare(m, ea, eb, rhs, invd, g, nx, ny);
}
void sweep_maps_prepare(LevelMaps* m, const DF32& ea, const DF32& eb, const DF32& rhs, const DF32& invd,
                        const Geo32& g, int nx, int ny) {
    prepare(m, ea, eb, rhs, invd, g, nx, ny);
}

bool sweep_fusable(const BCd& b) {
    for (int s = 0; s < 4; ++s) {
        const int t = b.type[s];
        if (t != T_DIRI && t != T_NEUM && t != T_PERIODIC) return false;
    }
    return true;
}

// The tiles of one sweep of a large level.  Away from the sides a tile needs 4
// columns left, 2 right and 4 rows either side of it (a column is reached
// through fewer colours than a row); beside a side, where the boundary pass
// reads two cells further, 6, 4, 6 and 6.  So the grid is cut into an inner
// rectangle of larger tiles and a frame of bands along the sides.
template <class T>
SweepTiles sweep_large_tiles(int nx, int ny) {
    using L = typename Shapes<T>::Large;
    constexpr int bx0 = L::WX - 4, bx1 = L::WX - 6, by = L::WY - 6;   // bands: left, right, bottom and top
    SweepTiles S = {};
    const auto add = [&](int x0, int x1, int y0, int y1, int tx, int ty, int inner) {
        SweepTiles::Region& R = S.r[S.n++];
        const int hx = (x1 - x0 + 1) / 2, hy = (y1 - y0 + 1) / 2;
        R.x0 = x0, R.x1 = x1, R.y0 = y0, R.y1 = y1, R.inner = inner;
        R.gx = (hx + tx / 2 - 1) / (tx / 2);
        R.gy = (hy + ty / 2 - 1) / (ty / 2);
        R.px = hx / R.gx, R.rx = hx % R.gx, R.py = hy / R.gy, R.ry = hy % R.gy;
        R.first = S.total;
        S.total += R.gx * R.gy;
    };
    if (nx < bx0 + bx1 + L::WX || ny < 2 * by + L::WY) {   // too narrow for a frame
        add(0, nx, 0, ny, nx <= L::WX ? L::WX : L::tx(1), ny <= L::WY ? L::WY : L::ty(1), 0);
        return S;
    }
    const int xr = (nx - bx1 + 1) & ~1, yt = (ny - by + 1) & ~1;   // even
    add(0, nx, 0, by, L::tx(1), by, 0);
    add(0, nx, yt, ny, L::tx(1), by, 0);
    add(0, bx0, by, yt, bx0, L::ty(1), 0);
    add(xr, nx, by, yt, bx1, L::ty(1), 0);
    add(bx0, xr, by, yt, L::WX - 6, L::WY - 8, 1);
    return S;
}
template SweepTiles sweep_large_tiles<float>(int, int);
template SweepTiles sweep_large_tiles<double>(int, int);

// Sweeps of the next launch, of `left` still to do.  A level inside one window
// takes all of them; a level whose tiles for 4 (2, 1) sweeps do not outnumber
// the SMs takes that many in the small shape, since its launch lasts one CTA's
// latency whatever it recomputes in the halo (256^2 in FP32: 2.3 us a sweep at
// 4, 3.0 at 2, 4.6 at 1; 512^2, where 4 and 2 need a second round: 7.0, 5.6 and
// 5.8).  A larger one takes one in the large shape (1024^2 in FP32: 13.0 us against
// 13.5 for two a launch, 2048^2: 36.7 against 48.1).  A caller's arrays (FP64), without
// descriptors, stay with the small shape, two sweeps a launch up to six rounds of
// its tiles: a pair shares one read of the operands, but a window of 32 x 48 holds
// 14 x 28 cells of a pair's tile and 22 x 36 of a single sweep's, so with many
// rounds the pair sweeps twice as many windows (us a sweep, pairs / singles, by the
// pairs' rounds: 384^2 at 2.6 9.3 / 11.5, 512^2 at 4.8 14.4 / 14.4, 577^2 at 6.0
// 17.5 / 18.4, 640^2 at 7.1 19.5 / 18.5, 1024^2 at 18.5 45 / 39, 2048^2 at 74
// 166 / 139).  A periodic side's ghosts come from global memory as they stand at
// the start of the launch, so it takes one.
template <class T>
SweepPlan sweep_plan(int nx, int ny, const BCd& b, int left, const LevelMaps* maps) {
    using S = typename Shapes<T>::Small;
    bool periodic = false;
    for (int s = 0; s < 4; ++s) periodic = periodic || b.type[s] == T_PERIODIC;
    if (nx <= S::WX && ny <= S::WY) return tiles_of<S>(nx, ny, periodic ? 1 : left);
    for (int k = periodic ? 1 : 4; k >= 1; k /= 2) {
        if (left < k || S::tx(k) < 12 || S::ty(k) < 12) continue;
        const SweepPlan p = tiles_of<S>(nx, ny, k);
        if ((long)p.gx * p.gy <= sm_count()) return p;
    }
    if (maps && maps->ok) return SweepPlan{1, 0, 0, false};
    const SweepPlan two = tiles_of<S>(nx, ny, 2);
    const bool pair = !periodic && left >= 2 && S::ty(2) >= 12 && (long)two.gx * two.gy <= 6L * sm_count();
    return pair ? two : tiles_of<S>(nx, ny, 1);
}

template <class T>
SweepPlan sweep_tiles(int nx, int ny, int k) {
    using S = typename Shapes<T>::Small;
    if (S::tx(k) < 12 || S::ty(k) < 12) return SweepPlan{0, 0, 0, true};
    return tiles_of<S>(nx, ny, k);
}
template SweepPlan sweep_tiles<float>(int, int, int);
template SweepPlan sweep_tiles<double>(int, int, int);
int sweep_wave() { return sm_count(); }

template SweepPlan sweep_plan<float>(int, int, const BCd&, int, const LevelMaps*);
template SweepPlan sweep_plan<double>(int, int, const BCd&, int, const LevelMaps*);

cudaError_t launch_sweep9(const DF& pin, const DF& pout, const DF& rhs, const DF& invd, const Geo& g, const BCd& b,
                          int homog, int nx, int ny, double omega, const SweepPlan& p, int dependent,
                          const LevelMaps* maps, int* status, cudaStream_t st) {
    return sweep_impl(pin, pout, rhs, invd, g, b, homog, nx, ny, omega, p, dependent, maps, status, st);
}
cudaError_t launch_sweep9(const DF32& pin, const DF32& pout, const DF32& rhs, const DF32& invd, const Geo32& g,
                          const BCd& b, int homog, int nx, int ny, double omega, const SweepPlan& p, int dependent,
                          const LevelMaps* maps, int* status, cudaStream_t st) {
    return sweep_impl(pin, pout, rhs, invd, g, b, homog, nx, ny, omega, p, dependent, maps, status, st);
}

template <class T>
cudaError_t launch_sweep9_jobs(const SweepJobT<T>* jobs, const int* pre, int njobs, int nblocks, int k, int small,
                               int flip, int* status, cudaStream_t st) {
    if (njobs < 1 || nblocks < 1) return cudaSuccess;
    using S = typename Shapes<T>::Small;
    using L = typename Shapes<T>::Large;
    cudaError_t e = sweep_kernels_init();
    if (e != cudaSuccess) return e;
    cudaLaunchAttribute at;
    if (small) {
        const cudaLaunchConfig_t cfg = config(dim3(nblocks), S::kThreads, 0, 1, &at, st);
        e = cudaLaunchKernelEx(&cfg, k_sweep9_jobs<S>, jobs, pre, njobs, k, flip);
    } else {
        const int ctas = std::min(nblocks, L::kMinBlocks * sm_count());
        const cudaLaunchConfig_t cfg = config(dim3(ctas), L::kThreads, Stage<L>::kSmem, 1, &at, st);
        e = cudaLaunchKernelEx(&cfg, k_sweep9_stream_jobs<L>, jobs, pre, njobs, nblocks, flip, status);
    }
    count_launch();
    return e;
}
template cudaError_t launch_sweep9_jobs<double>(const SweepJobT<double>*, const int*, int, int, int, int, int,
                                                int*, cudaStream_t);
template cudaError_t launch_sweep9_jobs<float>(const SweepJobT<float>*, const int*, int, int, int, int, int,
                                               int*, cudaStream_t);

}  // namespace mgp
